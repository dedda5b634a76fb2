"""FP64 plan: one arithmetic, whatever memory is free.  The digits of its tensor-core
products lie in memory of the arenas, so that an evaluation takes no more than they do
and its results are the same bits with the memory it needs as with all of it."""
import gc

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _evaluate():
    from spdepy_gb300.workloads import build_model, nonstationary_advection_diffusion
    w = nonstationary_advection_diffusion(M=30, N=30, T=24)
    mod = build_model(w, "fp64")
    mod._ensure_model()
    mod.plan.set_obs(w.idx)
    y = torch.as_tensor(np.random.default_rng(5).normal(size=len(w.idx))).cuda()
    torch.cuda.synchronize()
    f, jac = mod.plan.loglike(mod.canonical(w.par), y)
    return f, jac, torch.cuda.mem_get_info()[0], mod


def test_same_bits_with_little_memory():
    _evaluate()  # the context and its libraries
    gc.collect()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    f, jac, left, mod = _evaluate()
    taken = free - left
    del mod
    gc.collect()
    torch.cuda.empty_cache()
    hold = torch.empty(int(torch.cuda.mem_get_info()[0] - taken - (64 << 20)), dtype=torch.uint8, device="cuda")
    try:
        f2, jac2, _, _ = _evaluate()
    finally:
        del hold
        gc.collect()
        torch.cuda.empty_cache()
    assert f2 == f and np.array_equal(jac2, jac)
