"""Diagonal blocks and panel solves of the mixed factor at the edges of their tiles.

A spatial grid of at most 128 cells is one front, so its cell count is the width of
the separator: the grids below give blocks of every kind (a partial 16-column
panel, one full panel, a full 64-column block, a second block of one column, ...).
Checked through what the factor does, against the exported Q in FP64.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
U32 = 2.0 ** -24


def _model(M, N, T=1):
    from spdepy_gb300.grids import Grid
    from spdepy_gb300.spdes import spde_init
    t = np.arange(T, dtype=float) if T > 1 else None
    grid = Grid(np.arange(M, dtype=float), np.arange(N, dtype=float), t, None, 3)
    mod0 = spde_init("whittle-matern", grid.spatial(), ani=True, ha=False, bc=3) if T > 1 else None
    mod = spde_init("whittle-matern" if T == 1 else "advection-diffusion", grid, ani=True, ha=False, bc=3, mod0=mod0)
    return mod


@pytest.mark.parametrize("M,N,T", [(3, 3, 1), (4, 4, 1), (17, 1 + 1, 1), (7, 7, 1), (9, 7, 1), (8, 8, 1), (13, 5, 1), (10, 8, 1),
                                   (11, 9, 1), (16, 8, 1), (23, 19, 1), (9, 8, 5), (21, 17, 4)])
def test_factor_solve_and_draw(M, N, T):
    mod = _model(M, N, T)
    mod._assemble(mod.par)
    logdet = mod.plan.factor(False, 0.0)
    from spdepy_gb300.spdes import stencil_to_csr
    Q = stencil_to_csr(mod.grid, mod.plan.export_q().cpu().numpy()).toarray()
    n = Q.shape[0]
    # |d logdet| = |tr(Q^-1 dQ)|: the rounding of Q to FP32, and of L at every later block
    sens = U32 * np.abs(np.linalg.inv(Q) * Q).sum() * (1 if n <= 64 else n)
    assert abs(logdet - np.linalg.slogdet(Q)[1]) <= sens + 1e-11 * n
    # the unrefined solve is backward stable in FP32: ||b - Q x|| <= c n u ||Q|| ||x||
    b = torch.as_tensor(np.random.default_rng(1).normal(size=(n, 3)))
    x = mod.plan.solve(b, refine=0)[0].cpu().numpy()
    res = np.linalg.norm(b.numpy() - Q @ x, axis=0)
    assert (res <= 8 * n * U32 * np.linalg.norm(Q, 2) * np.linalg.norm(x, axis=0)).all()
    # x = P L^-T z has x^T Q x = z^T z, up to the error of L and of one triangular solve
    z = torch.as_tensor(np.random.default_rng(2).normal(size=n))
    d = mod.plan.sample(z).cpu().numpy()
    bound = 8 * n * U32 * np.linalg.norm(Q, 2) * (d @ d)
    assert abs(d @ Q @ d - float(z @ z)) <= bound
