"""Kernels launched as programmatic dependents are resident while their predecessor still
writes; only what a plan's set-up wrote may be promised unchanging (__restrict__) to them."""
import glob
import os
import re

from host_kernels import CSRC

SETUP = {"tasks", "fronts", "F", "rmap", "blist", "iperm", "amap", "src0", "src1", "maps"}


def test_only_set_up_data_is_restrict():
    seen = set()
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            text = f.read()
        for m in re.finditer(r"__global__ void[^{]*\{", text):
            if "chain_wait();" not in text[m.end():text.index("\n}\n", m.end())]:
                continue
            name = re.search(r"(\w+)\((?=const (?:Row|Gemm|Diag|Extend|Mirror|Emu)|Q)", m.group(0))
            seen.add(name.group(1))
            promised = set(re.findall(r"__restrict__ (\w+)", m.group(0)))
            assert promised <= SETUP, (name.group(1), promised - SETUP)
    assert {"potrf_kernel", "extend_kernel", "gemv_kernel", "zgather_kernel", "fwd_chain_kernel", "emu_gemm_kernel",
            "tc_pair_kernel"} <= seen
