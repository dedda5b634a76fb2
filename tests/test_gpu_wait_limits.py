"""Bounded waits of the FP64 plan's tensor-core products, and of an inversion that runs beside a solve:
with the limit at 1 ns they give up, the call reports it, and with the default limit
the same plan gives the results that it gave before."""
import ctypes

import numpy as np
import pytest
import torch

from spdepy_gb300 import _native as nat

pytestmark = pytest.mark.gpu


class Limit:
    def __init__(self, plan):
        self.h = plan.h

    def __enter__(self):
        nat.check(nat.lib().spde_plan_set_wait_limit(self.h, 1), self.h)

    def __exit__(self, *exc):
        nat.check(nat.lib().spde_plan_set_wait_limit(self.h, 0), self.h)


def test_fp64_products():
    from spdepy_gb300.workloads import build_model, nonstationary_advection_diffusion
    w = nonstationary_advection_diffusion(M=20, N=20, T=8)
    mod = build_model(w, "fp64")
    mod._assemble(w.par)
    plan, L = mod.plan, nat.lib()
    ld0 = plan.factor(False, 0.0)
    z0 = plan.selinv().cpu().numpy()
    prof = np.zeros(10, dtype=np.int64)
    L.spde_plan_read_profile(plan.h, None, None, None, 1)
    nat.check(L.spde_plan_set_profiling(plan.h, 1), plan.h)
    ld = ctypes.c_double()
    try:
        with Limit(plan):
            rc = L.spde_factor(plan.h, 0, 0.0, ctypes.byref(ld))
    finally:
        L.spde_plan_read_profile(plan.h, None, None, prof.ctypes.data, 1)
        L.spde_plan_set_profiling(plan.h, 0)
    assert prof[3] > 0  # products ran (and gave up)
    assert rc == 2 and b"timed out" in L.spde_last_error(plan.h)
    with pytest.raises(nat.SpdeError):
        plan.solve(torch.zeros(w.grid.n, dtype=torch.float64))  # no valid factor
    assert plan.factor(False, 0.0) == ld0
    with Limit(plan):
        with pytest.raises(nat.SpdeError, match="timed out"):
            plan.selinv()
    assert plan.factor(False, 0.0) == ld0
    assert np.array_equal(plan.selinv().cpu().numpy(), z0)


def test_inversion_beside_a_solve():
    """One front of 128 rows: its factorisation and its solves with two columns wait for nothing, its
    inversion has a product on the tensor cores."""
    from spdepy_gb300.grids import Grid
    from spdepy_gb300.spdes import spde_init
    grid = Grid(np.arange(16, dtype=float), np.arange(8, dtype=float), None, None, 3)
    mod = spde_init("whittle-matern", grid, ani=True, ha=False, bc=3)
    mod._ensure_model()
    plan, canon = mod.plan, mod.canonical(mod.par)
    plan.set_obs(np.arange(0, 128, 5))
    y = torch.as_tensor(np.random.default_rng(2).normal(size=(26, 2)))
    f0, jac0 = plan.loglike(canon, y)
    with Limit(plan):
        f1, _ = plan.loglike(canon, y, 0)  # no inversion: nothing waits
        assert f1 == f0
        with pytest.raises(nat.SpdeError, match="timed out"):
            plan.loglike(canon, y)
    f2, jac2 = plan.loglike(canon, y)
    assert f2 == f0 and np.array_equal(jac2, jac0)
