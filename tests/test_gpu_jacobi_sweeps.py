"""Damped Jacobi smoothing with few sweeps (its launches differ for one, an even and an odd number),
against the exported matrix."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 4])
@pytest.mark.parametrize("sweeps", [0, 1, 2, 3])
@pytest.mark.parametrize("nrhs", [1, 3])
def test_few_sweeps(T, sweeps, nrhs):
    from spdepy_gb300.grids import Grid
    from spdepy_gb300.spdes import spde_init, stencil_to_csr
    grid = Grid(np.arange(9.0), np.arange(7.0), np.arange(float(T)) if T > 1 else None, None, 3)
    mod0 = spde_init("whittle-matern", grid.spatial(), ani=True, ha=False, bc=3, precision="iterative") if T > 1 else None
    mod = spde_init("whittle-matern" if T == 1 else "advection-diffusion", grid, ani=True, ha=False, bc=3, mod0=mod0,
                    precision="iterative")
    mod._assemble(mod.par)
    n, tau, omega = grid.n, 2.0, 0.6
    mod.plan.set_obs(np.arange(0, n, 5))
    A = stencil_to_csr(grid, mod.plan.export_q(True, tau).cpu().numpy())
    z = np.random.default_rng(1).normal(size=(n, nrhs))
    ref, d = z.copy(), A.diagonal()[:, None]
    for _ in range(sweeps):
        ref = ref - omega * (A @ ref) / d
    ref /= np.sqrt((ref ** 2).mean(axis=0))
    got = torch.as_tensor(z).cuda().contiguous()
    mod.plan.jacobi_smooth(got, True, tau, omega, sweeps)
    # 43 products a sweep and the scaling, each entry of (I - omega D^-1 A) at most about 2 in sum
    assert np.abs(got.cpu().numpy() - ref).max() <= (sweeps + 1) * 2 ** sweeps * 64 * 2.0 ** -53 * np.abs(ref).max()
