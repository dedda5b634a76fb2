"""The gradient's sums over the cells, on grids one cell short of, at and one cell past the 512
cells that a cluster takes at a time, against the oracle's gradient with exact traces, for
25 coefficients per field (no multiple of the eight summed together)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(73, 7), (32, 16), (27, 19)])
def test_gradient_at_cluster_edges(M, N):
    from oracle.spde_oracle import OracleGrid, OracleModel
    from spdepy_gb300.workloads import build_model, nonstationary_advection_diffusion
    w = nonstationary_advection_diffusion(M=M, N=N, T=2)
    w.y = np.random.default_rng(0).normal(size=w.idx.size)
    og = OracleGrid(np.arange(float(M)), np.arange(float(N)), np.arange(2.0), None, 5)
    om = OracleModel(og, "cov-advection-var-diffusion", "ani", w.bc, ww=w.ww)
    om.derivative = "true"
    f0, j0 = om.loglike(w.par, w.y, w.idx, grad=True, exact=True)
    mod = build_model(w, "fp64")
    mod.initFit(w.y, idx=w.idx)
    f, j = mod.logLike(w.par, grad=True)
    # the sums run in FP64 on both sides; the solves and inverses leave 1e-10
    assert abs(f - f0) <= 1e-10 * abs(f0)
    assert np.abs(j - j0).max() <= 1e-8 * np.abs(j0).max()
