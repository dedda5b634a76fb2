"""FP64 plan: products from exact digit products on the tensor cores, at the edges of
their tiles, against dense FP64 algebra; infinities and NaN still end in an error (a parameter that is not finite is refused before)."""
import numpy as np
import pytest

from spdepy_gb300 import _native as nat

pytestmark = pytest.mark.gpu
U64 = 2.0 ** -53


def _spatial(M, N, kappa=-1.0):
    from spdepy_gb300.grids import Grid
    from spdepy_gb300.spdes import spde_init
    grid = Grid(np.arange(M, dtype=float), np.arange(N, dtype=float), None, None, 3)
    mod = spde_init("whittle-matern", grid, ani=True, ha=False, bc=3, precision="fp64")
    mod.par[0] = kappa
    return mod


@pytest.mark.parametrize("M,N", [(12, 12), (13, 17), (33, 8), (31, 33), (40, 27), (64, 20), (9, 65)])
@pytest.mark.parametrize("kappa", [0.5, -4.0])
def test_inverse_on_pattern(M, N, kappa):
    from spdepy_gb300.spdes import stencil_to_csr
    mod = _spatial(M, N, kappa)
    mod._assemble(mod.par)
    logdet = mod.plan.factor(False, 0.0)
    Q = stencil_to_csr(mod.grid, mod.plan.export_q().cpu().numpy()).toarray()
    n = Q.shape[0]
    ld = 2 * np.log(np.diag(np.linalg.cholesky(Q))).sum()  # slogdet's LU is off by 1e-14 relative itself
    cond = np.linalg.cond(Q)
    assert abs(logdet - ld) <= 8 * n * U64 * cond
    Z = mod.plan.selinv().cpu().numpy()[:, mod.plan.nslots // 2]
    ref = np.diag(np.linalg.inv(Q))
    # a backward-stable inverse: relative error below c n u cond
    assert np.abs(Z - ref).max() <= 8 * n * U64 * cond * np.abs(ref).max()


def test_overflow_is_reported():
    mod = _spatial(24, 24)
    par = mod.par.copy()
    mod._ensure_model()
    canon = mod.canonical(par)
    canon[1] = 800.0  # log gamma: exp overflows, stencil values are infinite or NaN
    mod.plan.assemble(canon)
    with pytest.raises(nat.NotPositiveDefiniteError):
        mod.plan.factor(False, 0.0)
    mod._assemble(par)  # the plan is usable afterwards
    assert np.isfinite(mod.plan.factor(False, 0.0))
