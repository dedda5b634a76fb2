"""PCG: how a solve's columns are grouped.  Two or three widths are as many launches of every
kernel, one after the other, which small solves with 3, 5, 7, ... columns do not repay."""
import ctypes

import pytest

from host_kernels import compile_host, section

TAIL = 'extern "C" int grouped(int64_t n, int nrhs) { return columns_grouped(n, nrhs); }'


@pytest.fixture(scope="module")
def lib():
    lib = compile_host([section("pcg.cu", "bool columns_grouped", "int pcg_solve")], TAIL)
    lib.grouped.argtypes = [ctypes.c_int64, ctypes.c_int]
    return lib


@pytest.mark.parametrize("n", [1920, 36000, 176000, 960000, 7680000])
def test_one_width_is_grouped(lib, n):
    assert all(lib.grouped(n, r) for r in (1, 2, 4, 8, 16, 200))


@pytest.mark.parametrize("n,nrhs,grouped", [(1920, 3, 0), (960000, 3, 0), (9600, 5, 0), (9600, 7, 0), (75600, 7, 0),
                                            (176000, 7, 0), (36000, 17, 1), (75600, 17, 1), (384000, 6, 1), (960000, 17, 1)])
def test_several_widths(lib, n, nrhs, grouped):
    assert lib.grouped(n, nrhs) == grouped
