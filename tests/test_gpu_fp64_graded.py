"""FP64 plan with parameter fields over several orders of magnitude: the inverse on the
pattern, entry by entry, relative to the standard deviations of its row and column, is as
close to the true one with products on the tensor cores as with FP64 FMAs (SPDE_TC=0, the
CUDA cores, in a process of its own)."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
# grid, logarithm of kappa (and gamma, where True) from -1 - a / 2 to -1 + a / 2
CASES = [((40, 30, 1), 9, False), ((15, 13, 9), 4, False), ((15, 13, 9), 10, False), ((20, 13, 7), 8, True), ((24, 9, 6), 12, False)]


def _model(shape, a, both):
    from spdepy_gb300.grids import Grid
    from spdepy_gb300.spdes import spde_init
    M, N, T = shape
    grid = Grid(np.arange(M, dtype=float), np.arange(N, dtype=float), np.arange(T, dtype=float) if T > 1 else None, None, 4)
    if T == 1:
        mod = spde_init("var-whittle-matern", grid, bc=3, precision="fp64")
    else:
        mod0 = spde_init("whittle-matern", grid.spatial(), ani=True, ha=False, bc=3, precision="fp64")
        mod = spde_init("advection-var-diffusion", grid, bc=3, mod0=mod0, precision="fp64")
    par, ramp = mod.par.copy(), np.linspace(-a / 2, a / 2, mod.layout.nk)
    par[mod.layout.sl["kappa"]] = -1 + ramp
    if both:
        par[mod.layout.sl["gamma"]] = -1 - ramp
    mod._assemble(par)
    return mod


def _inverses():
    out = []
    for case in CASES:
        mod = _model(*case)
        mod.plan.factor(False, 0.0)
        q = mod.plan.export_q().cpu().numpy()
        out.append((mod.grid, q, mod.plan.selinv().cpu().numpy()))
    return out


def _slices(X, axis):
    """X as a sum of four matrices whose products with each other are exact in FP64 (three of them)."""
    out = []
    for _ in range(3):
        top = np.abs(X).max(axis=axis, keepdims=True)
        s = 2.0 ** (np.ceil(np.log2(np.where(top > 0, top, 1))) + 33)
        out.append((X + s) - s)
        X = X - out[-1]
    return out + [X]


def _inverse(S):
    """S^-1 corrected twice by its residual in about 60 bits."""
    X = np.linalg.inv(S)
    for _ in range(2):
        a, b = _slices(S, 1), _slices(X, 0)
        R = np.eye(len(S)) - a[0] @ b[0]
        for i in range(4):
            for j in range(4):
                if 0 < i + j <= 4:
                    R = R - a[i] @ b[j]
        X = X + X @ R
    return X


def test_graded_fields(tmp_path):
    from spdepy_gb300.spdes import stencil_to_csr
    other = str(tmp_path / "z.npz")
    subprocess.run([sys.executable, os.path.abspath(__file__), other], check=True, env=dict(os.environ, SPDE_TC="0"))
    fma = np.load(other)
    for i, (grid, q, z) in enumerate(_inverses()):
        Q = stencil_to_csr(grid, q).toarray()
        d = 2.0 ** np.round(-0.5 * np.log2(np.diag(Q)))
        Z = _inverse(Q * d[:, None] * d) * d[:, None] * d
        sd = np.sqrt(np.diag(Z))
        err = []
        for v in (z, fma["z%d" % i]):
            v = stencil_to_csr(grid, v).tocoo()
            err.append(np.abs(v.data - Z[v.row, v.col]) / (sd[v.row] * sd[v.col]))
        assert np.sqrt(np.mean(err[0] ** 2)) <= 2 * np.sqrt(np.mean(err[1] ** 2)), CASES[i]  # one bit
        assert err[0].max() <= 4 * err[1].max(), CASES[i]


if __name__ == "__main__":
    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    np.savez(sys.argv[1], **{"z%d" % i: v[2] for i, v in enumerate(_inverses())})
