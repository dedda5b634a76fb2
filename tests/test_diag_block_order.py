"""Diagonal blocks: the result does not depend on which warp of the block runs first."""
import ctypes

import numpy as np
import pytest

from host_kernels import compile_host, section

TAIL = r"""
alignas(16) uint8_t potrf_sm[1 << 17];
struct Args { const DiagTask* t; double *L, *X, *lp; int* err; };
extern "C" void potrf_host(int w, int lda, double* L, double* X, double* lp, int* err, int up) {
  DiagTask t = {0, 0, lda, w, 7};
  Args a = {&t, L, X, lp, err};
  host::run({0, 0, 0}, {1, 1, 1}, 256, up, [](void* p) {
    Args* a = static_cast<Args*>(p);
    potrf_kernel<double>(a->t, a->L, a->X, a->lp, a->err);
  }, &a);
}
"""


@pytest.fixture(scope="module")
def lib():
    intc = section("kernels.cuh", "template <int N>\nstruct IntC", "enum GemmMode")
    task = section("kernels.cuh", "struct DiagTask", "// Extend-add task")
    kernel = section("dense.cu", "constexpr int kMaxNbk", "template <typename T>\nvoid launch_potrf")
    return compile_host([intc, task, kernel], TAIL)


@pytest.mark.parametrize("w", [1, 15, 16, 17, 31, 33, 48, 50, 64])
@pytest.mark.parametrize("up", [1, 0])
def test_factor_and_inverse(lib, w, up):
    g = np.random.default_rng(w).normal(size=(w, w))
    A = g @ g.T + w * np.eye(w)
    lda = w + 3
    L, X = np.full((w, lda), np.nan), np.full((64, 64), np.nan)
    L[:, :w] = np.tril(A)
    lp, err = np.zeros(1), np.full(1, -1, np.int32)
    lib.potrf_host(w, lda, *[v.ctypes.data_as(ctypes.c_void_p) for v in (L, X, lp, err)], up)
    ref = np.linalg.cholesky(A)
    tol = 8 * w * 2.0 ** -53 * np.linalg.cond(A)
    assert err[0] == -1
    assert np.abs(L[:, :w] - ref).max() <= tol * np.abs(ref).max()
    inv = np.linalg.inv(ref)
    assert np.abs(X[:w, :w] - inv).max() <= tol * np.abs(inv).max()
    assert abs(lp[0] - np.log(np.diag(ref)).sum()) <= tol * w


def test_first_column_is_rounded_once(lib):
    """The FP64 factor's first column, which no update reaches, is sqrt(a) and a_i / sqrt(a)."""
    rng = np.random.default_rng(9)
    for _ in range(40):
        w = 24
        A = np.diag(rng.uniform(0.5, 8.0, w)) + 0.0
        A[:, 0] += 1e-3 * rng.uniform(-1, 1, w)
        L, X = np.tril(A), np.zeros((64, 64))
        lp, err = np.zeros(1), np.full(1, -1, np.int32)
        lib.potrf_host(w, w, *[v.ctypes.data_as(ctypes.c_void_p) for v in (L, X, lp, err)], 1)
        root = np.sqrt(A[0, 0])
        assert L[0, 0] == root and X[0, 0] == 1 / root
        assert np.array_equal(L[1:, 0], A[1:, 0] / root)
