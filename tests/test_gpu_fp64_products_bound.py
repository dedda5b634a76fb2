"""The FP64 plan's tensor-core product by itself, against extended precision, within the bound
that its kernel states: per value of k 9.1 2^-64 of the operands' row scales, and one
rounding to FP64.  One digit or one pair of digits less does not stay within it."""
import ctypes

import numpy as np
import pytest
import torch

from spdepy_gb300 import _native as nat

pytestmark = pytest.mark.gpu
SYMBOL = "_ZN4spde15launch_emu_gemmEPKNS_8EmuSplitEiPKNS_7EmuTaskEiPKdS7_PdiPhPiP11CUstream_sty"
DIGITS = 8
CHUNK = DIGITS * 4096


class Split(ctypes.Structure):
    _fields_ = [(f, ctypes.c_int64) for f in ("src", "dst", "exp")] + [(f, ctypes.c_int32) for f in ("ld", "rows", "k", "nch", "buf")]


class Task(ctypes.Structure):
    _fields_ = [(f, ctypes.c_int64) for f in ("a", "b", "c", "a_step", "ea", "eb")] + [
        (f, ctypes.c_int32) for f in ("ldc", "m", "n", "k0", "k1")]


def _device(structs, kind):
    raw = np.frombuffer(bytes((kind * len(structs))(*structs)), np.uint8).copy()
    return torch.as_tensor(raw).cuda()


def _product(A, B, lda, ldb, ldc, mode, C):
    (m, k), n = A.shape, B.shape[0]
    nch = (k + 31) // 32
    splits, where, cursor = [], [], 0
    for buf, (rows, ld) in enumerate(((m, lda), (n, ldb))):
        tiles = (rows + 63) // 64
        exp = cursor + tiles * nch * CHUNK
        where.append((cursor, exp // 4))
        for r in range(0, rows, 64):
            splits.append(Split(r * ld, cursor + r // 64 * nch * CHUNK, exp // 4 + r, ld, min(64, rows - r), k, nch, buf))
        cursor = exp + tiles * 256
    (da, ea), (db, eb) = where
    tasks = [Task(da + i // 64 * nch * CHUNK, db + j // 64 * nch * CHUNK, i * ldc + j, nch * CHUNK if m - i > 64 else 0, ea + i, eb + j,
                  ldc, min(128, m - i), min(64, n - j), 0, nch) for j in range(0, n, 64) for i in range(0, m, 128)]

    def padded(X, ld):
        full = np.full((X.shape[0], ld), np.nan)
        full[:, :X.shape[1]] = X
        return torch.as_tensor(full).cuda()

    a, b, c = padded(A, lda), padded(B, ldb), padded(C, ldc)
    ds, dt = _device(splits, Split), _device(tasks, Task)
    scratch = torch.zeros(cursor, dtype=torch.uint8, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    fn = getattr(nat.lib(), SYMBOL)
    fn.restype = None
    P = ctypes.c_void_p
    fn.argtypes = [P, ctypes.c_int, P, ctypes.c_int, P, P, P, ctypes.c_int, P, P, P, ctypes.c_uint64]
    fn(ds.data_ptr(), len(splits), dt.data_ptr(), len(tasks), a.data_ptr(), b.data_ptr(), c.data_ptr(), mode, scratch.data_ptr(),
       err.data_ptr(), torch.cuda.current_stream().cuda_stream, 2 * 10 ** 9)
    torch.cuda.synchronize()
    assert err.item() == 0
    return c.cpu().numpy()[:, :n]


def _operands(kind, m, n, k, rng):
    A, B = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (n, k))
    if kind == "cancelling":  # every entry 2^-20 of its terms: its rounding does not hide the digits'
        h = k // 2
        A[:, h:2 * h] = A[:, :h] * (1 + 2.0 ** -20 * rng.uniform(-1, 1, (m, h)))
        B[:, h:2 * h] = -B[:, :h] * (1 + 2.0 ** -20 * rng.uniform(-1, 1, (n, h)))
        A[:, 2 * h:] = 0
    if kind == "graded":
        A *= 2.0 ** rng.integers(-10, 1, (m, k)) * 2.0 ** rng.integers(-300, 300, (m, 1))
        B *= 2.0 ** rng.integers(-40, 1, (n, k)) * 2.0 ** rng.integers(-300, 300, (n, 1))
    return A, B


@pytest.mark.parametrize("kind", ["uniform", "cancelling", "graded"])
@pytest.mark.parametrize("m,n,k", [(130, 70, 4), (64, 64, 31), (128, 64, 32), (130, 65, 33), (9, 8, 128), (65, 130, 129), (40, 30, 577)])
def test_product_bound(kind, m, n, k):
    rng = np.random.default_rng(m + k)
    A, B = _operands(kind, m, n, k, rng)
    C0 = rng.normal(size=(m, n))
    got = _product(A, B, k + 3, k + 2, n + 1, 1, C0)  # C = A B'
    ref = np.zeros((m, n), np.longdouble)
    for q in range(k):
        ref += np.longdouble(A[:, q:q + 1]) * np.longdouble(B[:, q])[None, :]
    scale = lambda X: 2.0 ** (np.floor(np.log2(np.abs(X).max(axis=1))) + 1)
    bound = 9.1 * k * np.longdouble(2) ** -64 * np.multiply.outer(scale(A), scale(B)) + np.longdouble(2) ** -53 * 1.01 * np.abs(ref)
    # what the reference itself may be off by (64 bits on x86, 113 elsewhere)
    bound += k * np.finfo(np.longdouble).eps * (np.abs(np.longdouble(A)) @ np.abs(np.longdouble(B)).T)
    assert (np.abs(got - ref) <= bound).all()


def test_updates_and_infinities():
    rng = np.random.default_rng(7)
    A, B, C = rng.uniform(-1, 1, (70, 40)), rng.uniform(-1, 1, (20, 40)), rng.normal(size=(70, 20))
    P = _product(A, B, 40, 40, 20, 1, C)
    assert np.array_equal(_product(A, B, 40, 40, 20, 0, C), C - P)
    assert np.array_equal(_product(A, B, 40, 40, 20, 2, C), -P)
    assert np.array_equal(_product(A, B, 40, 40, 20, 3, C), C + P)
    A[3, 5] = np.inf
    B[4, 6] = np.nan
    Q = _product(A, B, 40, 40, 20, 1, C)
    assert np.isnan(Q[3]).all() and np.isnan(Q[:, 4]).all()
    keep = np.ones((70, 20), bool)
    keep[3], keep[:, 4] = False, False
    assert np.array_equal(Q[keep], P[keep])
