"""PCG with every grouping of the right-hand sides (fours, a pair, single columns) on grids
whose rows and time steps are not multiples of a warp, against the exported matrix."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _plan(M, N, T, separable=False):
    from spdepy_gb300.grids import Grid
    from spdepy_gb300.spdes import spde_init
    t = np.arange(T, dtype=float) if T > 1 else None
    grid = Grid(np.arange(M, dtype=float), np.arange(N, dtype=float), t, None, 3)
    if separable:
        mod = spde_init("seperable-spatial-temporal", grid, ani=True, ha=False, bc=3, precision="mixed")
    else:
        mod0 = spde_init("whittle-matern", grid.spatial(), ani=True, ha=False, bc=3, precision="iterative") if T > 1 else None
        mod = spde_init("whittle-matern" if T == 1 else "advection-diffusion", grid, ani=True, ha=False, bc=3, mod0=mod0,
                        precision="iterative")
    mod._assemble(mod.par)
    return mod


@pytest.mark.parametrize("M,N,T", [(5, 4, 3), (31, 9, 2), (33, 17, 5), (64, 6, 3), (97, 3, 4), (40, 24, 1)])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 4, 6, 7, 9])
@pytest.mark.parametrize("precond", ["none", "jacobi", "learned", "per-node"])
def test_true_residual(M, N, T, nrhs, precond):
    from spdepy_gb300.precond import LearnedPreconditioner, init_params
    from spdepy_gb300.spdes import stencil_to_csr
    mod = _plan(M, N, T)
    n, plan = mod.grid.n, mod.plan
    rng = np.random.default_rng(n + nrhs)
    plan.set_obs(np.sort(rng.choice(n, max(1, n // 7), replace=False)))
    tau = 3.0
    A = stencil_to_csr(mod.grid, plan.export_q(True, tau).cpu().numpy())
    b = rng.normal(size=(n, nrhs))
    if nrhs > 1:
        b[:, 1] = 0.0  # a finished column from the start
    w, kind = None, precond
    if precond in ("learned", "per-node"):
        prm = init_params(3)
        prm[-27 * 33:] = 0.02 * rng.normal(size=27 * 33)
        w = LearnedPreconditioner(params=prm).weights(plan, True, tau, compact=precond == "learned")
        kind = "learned"
    tol = 1e-9
    x, it, rel = plan.pcg(torch.as_tensor(b), True, tau, kind, w=w, tol=tol, maxit=20000)
    x = x.cpu().numpy().reshape(n, nrhs)
    res = np.linalg.norm(b - A @ x, axis=0)
    assert (res <= tol * (1 + 1e-6) * np.linalg.norm(b, axis=0)).all()
    if nrhs > 1:
        assert not x[:, 1].any()


@pytest.mark.parametrize("M,N,T,nrhs", [(9, 7, 4, 1), (33, 5, 3, 3), (12, 11, 5, 6)])
def test_true_residual_separable(M, N, T, nrhs):
    from spdepy_gb300.spdes import stencil_to_csr
    mod = _plan(M, N, T, separable=True)
    n = mod.grid.n
    A = stencil_to_csr(mod.grid, mod.plan.export_q().cpu().numpy())
    b = np.random.default_rng(4).normal(size=(n, nrhs))
    x, _, _ = mod.plan.pcg(torch.as_tensor(b), False, 0.0, "jacobi", tol=1e-9, maxit=20000)
    res = np.linalg.norm(b - A @ x.cpu().numpy().reshape(n, nrhs), axis=0)
    assert (res <= 1e-9 * (1 + 1e-6) * np.linalg.norm(b, axis=0)).all()


@pytest.mark.parametrize("M,N,T,separable", [(8, 4, 3652, False), (11, 3, 3652, False), (11, 3, 3652, True),
                                             (8, 4, 3650, True), (129, 67, 105, False)])
def test_one_column_through_time(M, N, T, separable):
    """Long runs of time steps of a single column keep the coefficients in registers; the
    column's arithmetic is that of any other grouping, so the solutions are the same bits."""
    mod = _plan(M, N, T, separable=separable)
    n, plan = mod.grid.n, mod.plan
    rng = np.random.default_rng(n)
    plan.set_obs(np.sort(rng.choice(n, n // 7, replace=False)))
    b = torch.as_tensor(rng.normal(size=(n, 1)))
    one, it1, rel1 = plan.pcg(b, True, 3.0, "jacobi", tol=1e-9, maxit=20000)
    two, it2, rel2 = plan.pcg(b.repeat(1, 2), True, 3.0, "jacobi", tol=1e-9, maxit=20000)
    one, two = one.cpu().numpy().reshape(n), two.cpu().numpy().reshape(n, 2)
    assert it1 == it2
    assert np.isfinite(one).all() and one.any()
    assert np.array_equal(one, two[:, 0]) and np.array_equal(one, two[:, 1])
