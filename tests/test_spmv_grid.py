"""Launch shape of the FP64 stencil product: within the grid's limits and over every time step."""
import ctypes

import pytest

from host_kernels import compile_host, section

FAKE = """
struct QStencil { int Ns, T; };
struct dim3 { unsigned x, y, z; dim3(unsigned a, unsigned b) : x(a), y(b), z(1) {} };
static int nblk(int64_t n, int b) { return int((n + b - 1) / b); }
"""
TAIL = """
extern "C" void shape(int Ns, int T, int nrhs, int* out) {
  QStencil q = {Ns, T};
  const dim3 g = spmv_grid(q, nrhs, out);
  out[1] = g.x; out[2] = g.y;
}
"""


@pytest.fixture(scope="module")
def lib():
    return compile_host([FAKE, section("assemble.cu", "static dim3 spmv_grid", "void launch_spmv")], TAIL)


@pytest.mark.parametrize("Ns", [1, 4, 7, 300, 10000, 160000])
@pytest.mark.parametrize("T", [1, 2, 13, 48, 65535, 65537, 100000, 3000000])
@pytest.mark.parametrize("nrhs", [1, 4])
def test_shape(lib, Ns, T, nrhs):
    if Ns * T * nrhs >= 2 ** 31:
        pytest.skip("refused")
    out = (ctypes.c_int * 3)()
    lib.shape(Ns, T, nrhs, out)
    steps, x, y = out
    assert 1 <= y <= 65535 and y * steps >= T > (y - 1) * steps and x * 128 >= Ns * nrhs
