"""A solve with compact weights that has no memory for the rows of G^T next to observed nodes
looks their weights up, with the same result."""
import gc

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _solver(M, N, T, seed=3):
    from spdepy_gb300.grids import Grid
    from spdepy_gb300.precond import LearnedPreconditioner, init_params
    from spdepy_gb300.spdes import spde_init
    grid = Grid(*[np.arange(v, dtype=float) for v in (M, N, T)], None, 3)
    mod0 = spde_init("whittle-matern", grid.spatial(), ani=True, ha=False, bc=3, precision="iterative")
    mod = spde_init("advection-diffusion", grid, ani=True, ha=False, bc=3, mod0=mod0, precision="iterative")
    mod._assemble(mod.par)
    rng = np.random.default_rng(seed)
    mod.plan.set_obs(np.sort(rng.choice(grid.n, grid.n // 20, replace=False)))
    prm = init_params(3)
    prm[-27 * 33:] = 0.02 * rng.normal(size=27 * 33)
    w = LearnedPreconditioner(params=prm).weights(mod.plan, True, 2.0, compact=True)
    b = torch.as_tensor(rng.normal(size=grid.n)).cuda()
    torch.cuda.synchronize()
    return mod, lambda: mod.plan.pcg(b, True, 2.0, "learned", w=w, tol=1e-6, maxit=2000)


def test_same_solution_with_little_memory():
    M, N, T = 400, 400, 24
    n = M * N * T
    mod, solve = _solver(M, N, T)
    x, it, _ = solve()
    x = x.cpu()
    del mod, solve
    gc.collect()
    torch.cuda.empty_cache()
    mod, solve = _solver(M, N, T)
    # 26 floats a node and 69 a cell for the solve and its results, a third of it to spare; the rows take 27 a node
    keep = int(4 / 3 * 4 * (6 * n + n + 69 * M * N) + 4 * 8 * n)
    assert keep < 4 * 27 * n + 4 * 7 * n
    hold = torch.empty(torch.cuda.mem_get_info()[0] - keep, dtype=torch.uint8, device="cuda")
    try:
        x2, it2, _ = solve()
        x2 = x2.cpu()
    finally:
        del hold, mod, solve
        gc.collect()
        torch.cuda.empty_cache()
    assert it2 == it and torch.equal(x2, x)
