"""Workloads of the framework, through its public entry points, for timing and comparison.

Each case is one call that a user's program makes in earnest:

* ``fit``: one objective + exact gradient of a maximum-likelihood fit (``logLike(par, grad=True)``), the call every
  optimiser step makes, in the mixed plan (the default) and in the FP64 plan;
* ``predict``: the conditional mean and the marginal variances of the prediction loop (``Model.update``, ``Model.qinv``);
* ``draws``: a factorisation and a block of draws P L^-T z (``plan.factor``, ``plan.sample``);
* ``pcg``: solves on grids that are not factored (``plan.pcg``), one right-hand side (a conditional mean) or several (posterior
  draws, trace probes);
* ``train``: one training step of the learned preconditioner (assembly, weights, probes, gradient, Adam).

Models, parameters and observation patterns are those of ``spdepy_gb300/workloads.py`` (a non-stationary advection-diffusion with
a given velocity field, 5 x 5 B-splines and Dirichlet boundaries; a stationary one with Neumann boundaries) and the spatial
Whittle-Matern field of the reference's tutorials.  The data are a smooth moving field plus noise.
"""
import math

import numpy as np
import torch

NBS = 5          # B-splines per axis of the spatially varying models
PCG_TOL = 1e-8   # the default tolerance of plan.pcg


def listed():
    return [
        # the smallest grids people start with (tutorial size): an optimiser step is launches and latency
        {"name": "fit_small", "kind": "fit", "model": "stationary", "M": 16, "N": 16, "T": 8, "precision": "mixed", "obs": 0.2, "r": 1},
        # an odd, ragged grid of a pilot study
        {"name": "fit_ragged", "kind": "fit", "model": "nonstationary", "M": 47, "N": 39, "T": 13, "precision": "mixed", "obs": 0.01, "r": 1},
        # the stationary 100 x 100 x 24 configuration, 2,000 observations per time step
        {"name": "fit_stationary", "kind": "fit", "model": "stationary", "M": 100, "N": 100, "T": 24, "precision": "mixed", "obs": 0.2, "r": 1},
        # the headline configuration: 200 x 200 x 24, 107 parameters, 1 % observed
        {"name": "fit_headline", "kind": "fit", "model": "nonstationary", "M": 200, "N": 200, "T": 24, "precision": "mixed", "obs": 0.01, "r": 1},
        # the FP64 plan where results are checked against the CPU path (the sub-grid the CPU baseline runs)
        {"name": "fit_fp64", "kind": "fit", "model": "nonstationary", "M": 30, "N": 30, "T": 24, "precision": "fp64", "obs": 0.01, "r": 1},
        # ... and the largest grid a user would fit in FP64 throughout
        {"name": "fit_fp64_large", "kind": "fit", "model": "nonstationary", "M": 48, "N": 48, "T": 24, "precision": "fp64", "obs": 0.01, "r": 1},
        # a spatial field with several replicates of the data (several right-hand sides in the mean)
        {"name": "fit_spatial", "kind": "fit", "model": "spatial", "M": 301, "N": 203, "T": 1, "precision": "mixed", "obs": 0.05, "r": 4},
        # the prediction loop: new observations, conditional mean, marginal variances
        {"name": "predict", "kind": "predict", "model": "stationary", "M": 100, "N": 100, "T": 24, "precision": "mixed", "obs": 0.2, "r": 1},
        # 256 draws of the prior on the same grid (the samples per second of the benchmark)
        {"name": "draws", "kind": "draws", "model": "stationary", "M": 100, "N": 100, "T": 24, "precision": "mixed", "obs": 0.2, "r": 256},
        # a conditional mean on a grid that is not factored
        {"name": "pcg_mean", "kind": "pcg", "model": "nonstationary", "M": 400, "N": 400, "T": 48, "precision": "iterative", "obs": 0.01, "r": 1, "precond": "jacobi"},
        # posterior draws without a factor: many right-hand sides, the learned preconditioner
        {"name": "pcg_draws", "kind": "pcg", "model": "nonstationary", "M": 200, "N": 200, "T": 24, "precision": "iterative", "obs": 0.01, "r": 17, "precond": "learned"},
        # one training step of that preconditioner at its training size
        {"name": "train", "kind": "train", "model": "nonstationary", "M": 100, "N": 100, "T": 12, "precision": "iterative", "obs": 0.01, "r": 4},
    ]


def _spread(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit", "fit", "fit_fp64", "fit_spatial", "predict", "draws", "pcg", "pcg", "train"])
    model = rng.choice(["stationary", "nonstationary"])
    if kind == "fit":
        m = _spread(rng, 12, 180)
        return {"kind": "fit", "model": model, "M": m, "N": max(9, int(m * rng.uniform(0.6, 1.1))), "T": rng.randint(3, 24),
                "precision": "mixed", "obs": rng.choice([0.01, 0.05, 0.2]), "r": rng.choice([1, 1, 3])}
    if kind == "fit_fp64":
        m = _spread(rng, 10, 46)
        return {"kind": "fit", "model": model, "M": m, "N": max(9, int(m * rng.uniform(0.6, 1.0))), "T": rng.randint(3, 24),
                "precision": "fp64", "obs": rng.choice([0.01, 0.2]), "r": 1}
    if kind == "fit_spatial":
        m = _spread(rng, 20, 400)
        return {"kind": "fit", "model": "spatial", "M": m, "N": max(12, int(m * rng.uniform(0.4, 1.1))), "T": 1,
                "precision": rng.choice(["mixed", "mixed", "fp64"]), "obs": 0.05, "r": rng.choice([1, 4, 9])}
    if kind in ("predict", "draws"):
        m = _spread(rng, 14, 130)
        return {"kind": kind, "model": model, "M": m, "N": max(9, int(m * rng.uniform(0.6, 1.1))), "T": rng.randint(3, 24),
                "precision": "mixed", "obs": rng.choice([0.01, 0.2]), "r": 1 if kind == "predict" else rng.choice([1, 5, 64, 200])}
    if kind == "pcg":
        m = _spread(rng, 30, 300)
        return {"kind": "pcg", "model": model, "M": m, "N": max(12, int(m * rng.uniform(0.6, 1.1))), "T": rng.randint(3, 36),
                "precision": "iterative", "obs": rng.choice([0.01, 0.1]), "r": rng.choice([1, 1, 2, 9, 16]),
                "precond": rng.choice(["jacobi", "learned", "none"])}
    m = _spread(rng, 24, 130)
    return {"kind": "train", "model": "nonstationary", "M": m, "N": max(12, int(m * rng.uniform(0.6, 1.0))), "T": rng.randint(3, 14),
            "precision": "iterative", "obs": 0.01, "r": rng.choice([4, 4, 6])}


# ------------------------------------------------------------------ the inputs, from the seed alone
def _velocity(M, N, rng, modes=16, amplitude=0.5):
    """A smooth divergence-free velocity at the cells: a stream function of plane waves of 20 to 80 cells."""
    k = np.arange(M * N)
    we, wn = np.zeros(M * N), np.zeros(M * N)
    for _ in range(modes):
        lam, ang, ph = rng.uniform(20, 80), rng.uniform(0, 2 * np.pi), rng.uniform(0, 2 * np.pi)
        s = amplitude * math.sqrt(2 / modes) * np.sin(2 * np.pi / lam * (np.cos(ang) * (k % M) + np.sin(ang) * (k // M)) + ph)
        we, wn = we - np.sin(ang) * s, wn + np.cos(ang) * s
    return we, wn


def _inputs(case, seed):
    """Parameters, observation index, data, velocity and right-hand sides of a case (plain arrays)."""
    M, N, T, r = case["M"], case["N"], case["T"], case["r"]
    rng = np.random.default_rng(seed)
    n = M * N * T
    nb2 = NBS * NBS
    p = {"ww": None, "mod0": None}
    if case["model"] == "spatial":
        p["par"] = np.hstack([np.log(0.3) + rng.normal(0, 0.1, nb2), np.log(0.5) + rng.normal(0, 0.1, nb2), rng.normal(0, 0.3, nb2),
                              rng.normal(0, 0.3, nb2), np.log(1 / 0.1 ** 2)])
    else:
        p["mod0"] = np.array([np.log(0.3), np.log(0.5), np.sqrt(0.5), 0.05])
        if case["model"] == "stationary":
            p["par"] = np.hstack([np.log(0.3) + rng.normal(0, 0.05), np.log(0.5) + rng.normal(0, 0.05), np.sqrt(0.5), 0.1,
                                  0.3 + rng.normal(0, 0.02), -0.2 + rng.normal(0, 0.02), 0.0, p["mod0"], np.log(1 / 0.05 ** 2)])
        else:
            p["we"], p["wn"] = _velocity(M, N, rng)
            p["par"] = np.hstack([np.full(nb2, np.log(0.3)), np.full(nb2, np.log(0.5)), rng.normal(0, 0.3, nb2), rng.normal(0, 0.3, nb2),
                                  rng.uniform(0.7, 1.3), 0.0, p["mod0"], np.log(1 / 0.1 ** 2)])
    p["idx"] = np.sort(rng.choice(n, max(2, int(round(case["obs"] * n))), replace=False))
    # a smooth field that moves, plus noise, at the observed nodes
    k, t = p["idx"] % (M * N), p["idx"] // (M * N)
    y = np.zeros((p["idx"].size, r if case["kind"] in ("fit", "predict") else 1))
    for c in range(y.shape[1]):
        for _ in range(4):
            lam, ang, ph = rng.uniform(10, 60), rng.uniform(0, 2 * np.pi), rng.uniform(0, 2 * np.pi)
            y[:, c] += 0.5 * np.sin(2 * np.pi / lam * (np.cos(ang) * (k % M) + np.sin(ang) * (k // M)) + 0.2 * t + ph)
    y += 0.1 * rng.normal(size=y.shape)
    p["y"] = y[:, 0] if y.shape[1] == 1 else y
    p["tau"] = float(np.exp(p["par"][-1]))
    return p


def _device_block(seed, n, r, signs=False):
    """n x r normal (or +-1) values on the GPU, from the seed."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    if signs:
        return torch.randint(0, 2, (n, r), device="cuda", generator=g, dtype=torch.int8).double() * 2 - 1
    return torch.randn(n, r, dtype=torch.float64, device="cuda", generator=g)


def _net(seed):
    """A small preconditioner network: Glorot hidden layers, a last layer as training leaves it (small, nonzero)."""
    rng = np.random.default_rng(seed)
    shapes = [(32, 42), (32,), (32, 32), (32,), (27, 32), (27,)]
    parts = [(rng.normal(0, np.sqrt(1 / s[1]), s) if len(s) == 2 and s[0] == 32 else rng.normal(0, 0.01, s)).ravel() for s in shapes]
    return np.concatenate(parts).astype(np.float32)


def _rhs(case, seed, p):
    """Right-hand sides of a pcg case: tau S^T y for the mean, normal columns for the others."""
    n = case["M"] * case["N"] * case["T"]
    b = torch.zeros(n, dtype=torch.float64, device="cuda")
    b[torch.as_tensor(p["idx"]).cuda()] = torch.as_tensor(p["tau"] * p["y"]).cuda()
    if case["r"] == 1:
        return b
    return torch.cat([_device_block(seed, n, case["r"] - 1), b[:, None]], 1).contiguous()


def prepare(case, seed):
    from spdepy_gb300.grids import Grid
    from spdepy_gb300.model import Model
    from spdepy_gb300.spdes import spde_init
    M, N, T = case["M"], case["N"], case["T"]
    p = _inputs(case, seed)
    t = np.arange(T, dtype=float) if T > 1 else None
    grid = Grid(np.arange(M, dtype=float), np.arange(N, dtype=float), t, None, 3 if case["model"] == "stationary" else NBS)
    s = {"case": case, "p": p}
    prec = case["precision"]
    fam = {"spatial": "var-whittle-matern", "stationary": "advection-diffusion", "nonstationary": "cov-advection-var-diffusion"}[case["model"]]
    opts = {"ani": True, "ha": False, "bc": 1 if case["model"] == "stationary" else 3}
    mod0 = None if T == 1 else spde_init("whittle-matern", grid.spatial(), precision=prec, **opts)
    model = Model(spde=fam, grid=grid, mod0=mod0, precision=prec, **opts)
    mod = model.mod
    if case["model"] == "nonstationary":
        mod.initFit(p["y"], idx=p["idx"], ww=grid.assimilate_adv(p["we"], p["wn"]))
    mod.setPars(p["par"])
    s["model"], s["mod"] = model, mod
    plan = mod.plan
    kind = case["kind"]
    if kind == "fit":
        mod.initFit(p["y"], idx=p["idx"])
    elif kind == "predict":
        mod.setQ(p["par"])
    elif kind == "draws":
        s["z"] = _device_block(seed, grid.n, case["r"])
    elif kind == "pcg":
        mod._assemble(p["par"])
        plan.set_obs(p["idx"])
        s["b"] = _rhs(case, seed, p)
        if case["precond"] == "learned":
            from spdepy_gb300.precond import LearnedPreconditioner
            s["precond"] = LearnedPreconditioner(params=_net(7))
    elif kind == "train":
        plan.set_obs(p["idx"])
        s["z"] = _device_block(seed, grid.n, case["r"], signs=True)
        s["params"] = torch.as_tensor(_net(seed)).cuda()
    return s


def run(s):
    case, p, mod = s["case"], s["p"], s["mod"]
    kind, plan = case["kind"], mod.plan
    if kind == "fit":
        f, jac = mod.logLike(p["par"], grad=True)
        return {"f": f, "jac": jac}
    if kind == "predict":
        m = s["model"]
        m.setModel()
        m.update(p["y"], p["idx"])
        return {"mu": m.mu, "var": m.qinv()}
    if kind == "draws":
        mod._assemble(p["par"])
        logdet = plan.factor(False, 0.0)
        return {"logdet": logdet, "x": plan.sample(s["z"])}
    if kind == "pcg":
        w = s["precond"].weights(plan, True, p["tau"]) if case["precond"] == "learned" else None
        x, _, _ = plan.pcg(s["b"], True, p["tau"], case["precond"], w=w, tol=PCG_TOL, maxit=5000)
        return {"x": x}
    # one step of LearnedPreconditioner.train from fresh Adam moments
    mod._assemble(p["par"])
    prm, half = s["params"].clone(), case["r"] // 2
    w, act = plan.precond_weights(prm, True, p["tau"], keep_activations=True)
    zs = plan.jacobi_smooth(s["z"][:, :half].contiguous(), True, p["tau"], 0.6, 20)
    z = torch.cat([zs, s["z"][:, half:]], 1).contiguous()
    loss, grad = plan.precond_grad(prm, w, act, z, True, p["tau"])
    plan.adam_step(prm, grad, torch.zeros_like(prm), torch.zeros_like(prm), 1, lr=3e-3)
    return {"loss": loss, "grad": grad, "params": prm}


def work(case):
    from spdepy_gb300._native import symbolic_info
    M, N, T, r, kind = case["M"], case["N"], case["T"], case["r"], case["kind"]
    n = M * N * T
    m = max(2, int(round(case["obs"] * n)))
    stencil = 8 * 59 * M * N   # the assembled operator's coefficients
    if kind in ("fit", "predict", "draws"):
        info = symbolic_info(M, N, T)
        if kind == "fit":    # two factorisations, two selected inversions
            return {"bytes": 16 * m * r + stencil, "flops": 2 * info.factor_flops + 2 * info.selinv_flops}
        if kind == "predict":
            return {"bytes": 16 * m + 12 * n + stencil, "flops": 2 * info.factor_flops + info.selinv_flops}
        return {"bytes": 16 * n * r + stencil, "flops": info.factor_flops + 2 * info.nnz_l * r}
    if kind == "pcg":        # each right-hand side read, each solution written; the products of about 100 iterations
        return {"bytes": 16 * n * r + stencil, "flops": 100 * r * n * (2 * 43 + 10 + (4 * 27 if case["precond"] == "learned" else 0))}
    net = 42 * 32 + 32 * 32 + 27 * 32
    return {"bytes": 8 * n * r + stencil + 3 * 4 * 3323, "flops": n * (6 * net + r * (2 * 2 * 43 + 4 * 2 * 27 + 2 * 27 * 2) + r // 2 * 20 * 90)}


# ------------------------------------------------------------------ the same in 64 bits, in plain torch
def _bsplines(t, lo, hi):
    """Degree-2 B-splines, NBS of them on [lo, hi], the two end functions of each side merged."""
    kv = np.linspace(lo - 2 * (hi - lo) / NBS, hi + 2 * (hi - lo) / NBS, NBS + 5)
    B = np.stack([((t >= kv[i]) & (t < kv[i + 1])) * 1.0 for i in range(NBS + 4)], 1)
    for d in (1, 2):
        B = np.stack([(t - kv[i]) / (kv[i + d] - kv[i]) * B[:, i] + (kv[i + d + 1] - t) / (kv[i + d + 1] - kv[i + 1]) * B[:, i + 1]
                      for i in range(NBS + 4 - d)], 1)
    return np.hstack([(B[:, 0] + B[:, 1])[:, None], B[:, 2:-2], (B[:, -2] + B[:, -1])[:, None]])


def _basis(M, N, dx, dy):
    e = 0.5 if dx or dy else 0.0
    bx, by = _bsplines(np.arange(M) + dx, -e, M - 1 + e), _bsplines(np.arange(N) + dy, -e, N - 1 + e)
    b = by[:, None, :, None] * bx[None, :, None, :]   # y, x, by, bx
    return torch.as_tensor(b.reshape(N * M, NBS * NBS)).to(_dev())


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Spatial:
    """Nine-point operators on the M x N cells (unit spacing): coefficient fields c[(di, dj)] of shape (N, M)."""

    def __init__(self, M, N, neumann):
        self.M, self.N, self.neumann = M, N, neumann
        j, i = torch.meshgrid(torch.arange(N, device=_dev()), torch.arange(M, device=_dev()), indexing="ij")
        self.i, self.j = i, j

    def collect(self, entries):
        """Sum of entries {(di, dj): field}; an entry that leaves the grid is dropped (Dirichlet), or taken to the clamped cell."""
        c = {}
        for (di, dj), v in entries.items():
            ii, jj = self.i + di, self.j + dj
            inx, iny = (ii >= 0) & (ii < self.M), (jj >= 0) & (jj < self.N)
            if not self.neumann:
                parts = [((di, dj), v * (inx & iny))]
            else:
                parts = [((di, dj), v * (inx & iny)), ((0, dj), v * (~inx & iny)), ((di, 0), v * (inx & ~iny)), ((0, 0), v * (~inx & ~iny))]
            for k, w in parts:
                c[k] = c[k] + w if k in c else w
        return c

    def diffusion(self, W00, E00, N01, S01, N11, S11, E10, W10):
        if self.neumann:   # no flux through the boundary faces
            left, right, bot, top = self.i == 0, self.i == self.M - 1, self.j == 0, self.j == self.N - 1
            W00, W10, E00, E10 = W00 * ~left, W10 * ~left, E00 * ~right, E10 * ~right
            S11, S01, N11, N01 = S11 * ~bot, S01 * ~bot, N11 * ~top, N01 * ~top
        q = 0.25
        return self.collect({(0, 0): -(E00 + W00) - (N11 + S11), (1, 0): E00 + q * (N01 - S01), (-1, 0): W00 - q * (N01 - S01),
                             (0, 1): N11 + q * (E10 - W10), (0, -1): S11 - q * (E10 - W10), (1, 1): q * (N01 + E10),
                             (-1, -1): q * (S01 + W10), (-1, 1): -q * (N01 + W10), (1, -1): -q * (S01 + E10)})

    def advection_const(self, w0, w1):
        one = torch.ones(self.N, self.M, dtype=torch.float64, device=_dev())
        a0, a1 = w0.abs(), w1.abs()
        ctr = (a0 + a1) * one
        if self.neumann:
            ctr = ctr - a0 / 2 * ((self.i == 0).double() + (self.i == self.M - 1)) - a1 / 2 * ((self.j == 0).double() + (self.j == self.N - 1))
        c = {(0, 0): ctr, (1, 0): -(a0 - w0) / 2 * one * (self.i < self.M - 1), (-1, 0): -(a0 + w0) / 2 * one * (self.i > 0),
             (0, 1): -(a1 - w1) / 2 * one * (self.j < self.N - 1), (0, -1): -(a1 + w1) / 2 * one * (self.j > 0)}
        return c

    def advection_faces(self, E, Nn, W, S):
        aE, aN, aW, aS = E.abs(), Nn.abs(), W.abs(), S.abs()
        return self.collect({(0, 0): (aE + E + aW - W) / 2 + (aN + Nn + aS - S) / 2, (1, 0): -(aE - E) / 2, (-1, 0): -(aW + W) / 2,
                             (0, 1): -(aN - Nn) / 2, (0, -1): -(aS + S) / 2})

    def dense(self, c):
        n = self.M * self.N
        k = (self.j * self.M + self.i).reshape(-1)
        A = torch.zeros(n * n, dtype=torch.float64, device=_dev())
        for (di, dj), v in c.items():
            v = v.reshape(-1)
            ok = ((self.i + di >= 0) & (self.i + di < self.M) & (self.j + dj >= 0) & (self.j + dj < self.N)).reshape(-1)
            A = A.index_add(0, (k * n + k + dj * self.M + di)[ok], v[ok])
        return A.reshape(n, n)

    def shift(self, x, di, dj):
        """x at (i + di, j + dj), zero outside; x (..., N, M)."""
        out = torch.zeros_like(x)
        M, N = self.M, self.N
        out[..., max(0, -dj):N - max(0, dj), max(0, -di):M - max(0, di)] = x[..., max(0, dj):N - max(0, -dj), max(0, di):M - max(0, -di)]
        return out

    def apply(self, c, x):
        return sum(v * self.shift(x, di, dj) for (di, dj), v in c.items())

    def apply_t(self, c, x):
        return sum(self.shift(v * x, -di, -dj) for (di, dj), v in c.items())


def _operators(case, p, par):
    """(op, A, Qs, A0, scale): the coefficient fields of A and A0 and diag(Qs), differentiable in par."""
    M, N = case["M"], case["N"]
    op = _Spatial(M, N, case["model"] == "stationary")
    one = torch.ones(N, M, dtype=torch.float64, device=_dev())

    def const_wm(lk, lg, vx, vy):
        g = lg.exp()
        h00, h01, h11 = (g + vx * vx) * one, vx * vy * one, (g + vy * vy) * one
        return lk.exp() * one, op.diffusion(h00, h00, h01, h01, h11, h11, h01, h01)

    def field_wm(lk, lg, vx, vy):
        face = {}
        for key, d in (("W", (-0.5, 0.0)), ("E", (0.5, 0.0)), ("S", (0.0, -0.5)), ("N", (0.0, 0.5))):
            B = _basis(M, N, *d)
            g, a, b = (B @ lg).exp(), B @ vx, B @ vy
            face[key] = [(g + a * a).reshape(N, M), (a * b).reshape(N, M), (g + b * b).reshape(N, M)]
        kap = (_basis(M, N, 0.0, 0.0) @ lk).exp().reshape(N, M)
        return kap, op.diffusion(face["W"][0], face["E"][0], face["N"][1], face["S"][1], face["N"][2], face["S"][2], face["E"][1], face["W"][1])

    nb = NBS * NBS
    neg = lambda c: {k: -v for k, v in c.items()}
    plus = lambda c, k, v: {**c, k: c[k] + v}
    if case["model"] == "spatial":
        kap, D = field_wm(par[:nb], par[nb:2 * nb], par[2 * nb:3 * nb], par[3 * nb:4 * nb])
        return op, plus(neg(D), (0, 0), kap), None, None, None
    if case["model"] == "stationary":
        kap, D = const_wm(par[0], par[1], par[2], par[3])
        w, o = op.advection_const(par[4], par[5]), 6
    else:
        kap, D = field_wm(par[:nb], par[nb:2 * nb], par[2 * nb:3 * nb], par[3 * nb:4 * nb])
        we, wn = (torch.as_tensor(p[k].reshape(N, M)).to(_dev()) for k in ("we", "wn"))
        cl = lambda a, di, dj: a[(torch.arange(N, device=a.device) + dj).clamp(0, N - 1)][:, (torch.arange(M, device=a.device) + di).clamp(0, M - 1)]
        lam, o = par[4 * nb], 4 * nb + 1
        w = op.advection_faces(lam * (we + cl(we, 1, 0)) / 2, lam * (wn + cl(wn, 0, 1)) / 2, lam * (we + cl(we, -1, 0)) / 2, lam * (wn + cl(wn, 0, -1)) / 2)
    sigma, m0 = par[o].exp(), par[o + 1:o + 5]
    kap0, D0 = const_wm(m0[0], m0[1], m0[2], m0[3])
    A = plus(neg(D), (0, 0), 1.0 + kap)
    for k, v in w.items():
        A = plus(A, k, v)
    return op, A, kap * kap, plus(neg(D0), (0, 0), kap0), 1.0 / sigma


def _q_blocks(case, p, par):
    """Dense (first, middle, last) diagonal blocks and the off-diagonal block (t, t + 1) of Q."""
    op, A, qs, A0, sc = _operators(case, p, par)
    Ad = op.dense(A)
    if case["T"] == 1:
        return Ad.T @ Ad, None, None, None
    q = qs.reshape(-1)
    A0d = op.dense(A0)
    mid = Ad.T @ (q[:, None] * Ad) * sc
    D = torch.diag(q) * sc
    return A0d.T @ A0d + D, mid + D, mid, -(q[:, None] * Ad) * sc


def _posterior(case, p, blocks, inverse=True):
    """log det and (with inverse) the diagonal and upper off-diagonal blocks of the inverse of the block-tridiagonal matrix."""
    D0, Dm, Dl, O = blocks
    T, ns = case["T"], case["M"] * case["N"]

    def sweep(extra, b=None):
        Ls, ld, prev = [], 0.0, None
        for t in range(T):
            S = (D0 if t == 0 else Dl if t == T - 1 else Dm).clone()
            if extra is not None:
                S.diagonal().add_(extra[t])
            if prev is not None:
                S -= prev.T @ prev
            L = torch.linalg.cholesky(S)
            ld = ld + 2 * L.diagonal().log().sum()
            prev = torch.linalg.solve_triangular(L, O, upper=False) if t + 1 < T else None
            Ls.append(L)
        mu = None
        if b is not None:
            z, mu = [], [None] * T
            for t in range(T):
                r = b[t] - (O.T @ torch.cholesky_solve(z[-1], Ls[t - 1]) if t else 0.0)
                z.append(r)
            for t in range(T - 1, -1, -1):
                mu[t] = torch.cholesky_solve(z[t] - (O @ mu[t + 1] if t + 1 < T else 0.0), Ls[t])
        if not inverse:
            return ld, mu, None, None
        Zd, Zo = [None] * T, [None] * T
        for t in range(T - 1, -1, -1):
            Si = torch.cholesky_inverse(Ls[t])
            if t == T - 1:
                Zd[t] = Si
            else:
                U = Si @ O
                Zo[t] = -U @ Zd[t + 1]
                Zd[t] = Si - Zo[t] @ U.T
        return ld, mu, Zd, Zo

    return sweep, T, ns


def _exact_fit(case, p):
    par = torch.as_tensor(p["par"]).to(_dev()).requires_grad_()
    T, ns, r = case["T"], case["M"] * case["N"], case["r"]
    blocks = _q_blocks(case, p, par)
    plain = tuple(None if b is None else b.detach() for b in blocks)
    sweep, _, _ = _posterior(case, p, plain)
    tau, m = p["tau"], p["idx"].size
    hits = torch.zeros(T * ns, dtype=torch.float64, device=_dev())
    idx = torch.as_tensor(p["idx"]).to(_dev())
    hits[idx] = 1.0
    Y = torch.as_tensor(p["y"].reshape(m, r)).to(_dev())
    b = torch.zeros(T * ns, r, dtype=torch.float64, device=_dev())
    b[idx] = tau * Y
    ld, _, Zd, Zo = sweep(None)
    ldc, mu, Cd, Co = sweep(tau * hits.reshape(T, ns), b.reshape(T, ns, r))
    D0, Dm, Dl, O = plain
    quad = 0.0
    for t in range(T):
        Dt = D0 if t == 0 else Dl if t == T - 1 else Dm
        quad = quad + (mu[t] * (Dt @ mu[t])).sum() + (2 * (mu[t] * (O @ mu[t + 1])).sum() if t + 1 < T else 0.0)
    rss = ((Y - torch.cat(mu)[idx]) ** 2).sum()
    like = 0.5 * r * (ld - ldc) + m * r * math.log(tau) / 2 - 0.5 * quad - tau / 2 * rss
    G = [0.0, 0.0, 0.0, 0.0]   # d like / d (first, middle, last, off)
    for t in range(T):
        k = 0 if t == 0 else 2 if t == T - 1 else 1
        G[k] = G[k] + 0.5 * r * (Zd[t] - Cd[t]) - 0.5 * mu[t] @ mu[t].T
        if t + 1 < T:
            G[3] = G[3] + r * (Zo[t] - Co[t]) - mu[t] @ mu[t + 1].T
    s = sum((g * q).sum() for g, q in zip(G, blocks) if torch.is_tensor(g) and q is not None)
    g = torch.autograd.grad(s, par)[0]
    g[-1] = m * r / 2 - 0.5 * r * tau * (torch.cat([c.diagonal() for c in Cd]) * hits).sum() - tau / 2 * rss
    return {"f": -float(like) / (m * r), "jac": (-g / (m * r)).cpu().numpy()}


def _exact_linear(case, p):
    """x -> A x with A = Q + tau S^T S for x of shape (r, T, N, M), from the coefficient fields; and diag(A)."""
    par = torch.as_tensor(p["par"]).to(_dev())
    op, A, qs, A0, sc = _operators(case, p, par)
    T, N, M = case["T"], case["N"], case["M"]
    obs = torch.zeros(T * N * M, dtype=torch.float64, device=_dev())
    obs[torch.as_tensor(p["idx"]).to(_dev())] = p["tau"]
    obs = obs.reshape(T, N, M)

    def mul(x):
        e = op.apply(A, x[:, 1:]) - x[:, :-1]          # innovations
        out = obs * x
        out[:, 1:] += op.apply_t(A, qs * e) * sc
        out[:, :-1] -= qs * e * sc
        out[:, 0] += op.apply_t(A0, op.apply(A0, x[:, 0]))
        return out

    def diag():
        sq = lambda c, w: sum(op.shift(w * v * v, -di, -dj) for (di, dj), v in c.items())
        d = obs.clone()
        d[1:] += sq(A, qs) * sc
        d[:-1] += qs * sc
        d[0] += sq(A0, torch.ones_like(qs))
        return d

    return op, A, qs, A0, sc, obs, mul, diag


def _exact_pcg(case, seed, p):
    n, r = case["M"] * case["N"] * case["T"], case["r"]
    _, _, _, _, _, _, mul, diag = _exact_linear(case, p)
    shape = (r, case["T"], case["N"], case["M"])
    B = _rhs(case, seed, p).reshape(n, r).T.contiguous()
    X = torch.zeros_like(B)
    di = 1 / diag()
    dot = lambda a, b: (a * b).flatten(1).sum(1).reshape(-1, 1, 1, 1)
    for c in range(0, r, 4):   # four columns at a time
        b = B[c:c + 4].reshape(-1, *shape[1:])
        x, res = torch.zeros_like(b), b.clone()
        z = di * res
        q, rz, nb = z.clone(), dot(res, z), dot(b, b)
        for it in range(2000):
            aq = mul(q)
            al = rz / dot(q, aq)
            x += al * q
            res -= al * aq
            if it % 10 == 0 and bool((dot(res, res) <= 1e-26 * nb).all()):
                break
            z = di * res
            new = dot(res, z)
            q = z + new / rz * q
            rz = new
        X[c:c + 4] = x.reshape(x.shape[0], n)
    X = X.T.contiguous()
    return {"x": X[:, 0].contiguous() if r == 1 else X}


def _exact_train(case, seed, p):
    T, N, M, r = case["T"], case["N"], case["M"], case["r"]
    n = T * N * M
    op, A, qs, A0, sc, obs, mul, diag = _exact_linear(case, p)
    d = diag()
    # the 43 entries of every row: products of A with A on the nine points, by the coefficient fields
    off = [(dx, dy, dt) for dt, w in ((-1, 1), (0, 2), (1, 1)) for dy in range(-w, w + 1) for dx in range(-w, w + 1)]
    rows = {o: torch.zeros(T, N, M, dtype=torch.float64, device=_dev()) for o in off}

    def gram(c, w):   # (c^T diag(w) c) at offset o: sum over a of c_a(k - a) w(k - a) c_b(k - a), b = a + o
        g = {}
        for (ai, aj), u in c.items():
            for (bi, bj), v in c.items():
                o = (bi - ai, bj - aj)
                t = op.shift(u * w * v, -ai, -aj)
                g[o] = g[o] + t if o in g else t
        return g

    for (dx, dy), v in gram(A, qs).items():
        rows[(dx, dy, 0)][1:] += v * sc
    for (dx, dy), v in gram(A0, torch.ones_like(qs)).items():
        rows[(dx, dy, 0)][0] += v
    rows[(0, 0, 0)][:-1] += qs * sc
    rows[(0, 0, 0)] += obs
    for (dx, dy), v in A.items():
        rows[(dx, dy, 1)][:-1] -= qs * v * sc
        rows[(-dx, -dy, -1)][1:] -= op.shift(qs * v, -dx, -dy) * sc
    feat = torch.stack([rows[o].reshape(-1) / d.reshape(-1) for o in off if o != (0, 0, 0)], 1)
    s = d.reshape(-1).rsqrt()
    prm = torch.as_tensor(_net(seed)).to(_dev()).double().requires_grad_()
    cut, o = [], 0
    for shape in [(32, 42), (32,), (32, 32), (32,), (27, 32), (27,)]:
        k = int(np.prod(shape))
        cut.append(prm[o:o + k].reshape(shape))
        o += k
    h = torch.tanh(torch.tanh(feat @ cut[0].T + cut[1]) @ cut[2].T + cut[3]) @ cut[4].T + cut[5]
    w = h * s[:, None] + torch.nn.functional.one_hot(torch.tensor(13), 27).to(h) * s[:, None]
    w = w.T.reshape(27, T, N, M)

    def move(x, dx, dy, dt):
        out = torch.zeros_like(x)
        out[:, max(0, -dt):T - max(0, dt)] = op.shift(x, dx, dy)[:, max(0, dt):T - max(0, -dt)]
        return out

    offs = [(k % 3 - 1, (k // 3) % 3 - 1, k // 9 - 1) for k in range(27)]
    Gx = lambda x: sum(w[k] * move(x, *o) for k, o in enumerate(offs))
    Gt = lambda x: sum(move(w[k] * x, -o[0], -o[1], -o[2]) for k, o in enumerate(offs))
    z = _device_block(seed, n, r, signs=True).T.reshape(r, T, N, M).to(_dev())
    zs = z[:r // 2].clone()
    for _ in range(20):
        zs = zs - 0.6 * mul(zs) / d
    zs = zs / zs.flatten(1).square().mean(1).sqrt().reshape(-1, 1, 1, 1)
    z = torch.cat([zs, z[r // 2:]])
    e = z - Gx(mul(Gt(z)))
    loss = (e * e).sum() / (n * r)
    g = torch.autograd.grad(loss, prm)[0]
    return {"loss": float(loss.detach()), "grad": g, "params": (prm - 3e-3 * g / (g.abs() + 1e-8)).detach()}


def exact(case, seed):
    kind, ns, T = case["kind"], case["M"] * case["N"], case["T"]
    p = _inputs(case, seed)
    if kind == "pcg":
        return _exact_pcg(case, seed, p) if ns * T * case["r"] <= 17_000_000 else None
    if kind == "train":
        return _exact_train(case, seed, p)
    if ns ** 3 * T > 2 * 2500 ** 3 * 24 or ns > 8000:   # over about 20 seconds of dense 64-bit blocks
        return None
    if kind == "fit":
        return _exact_fit(case, p)
    plain = tuple(None if b is None else b.detach() for b in _q_blocks(case, p, torch.as_tensor(p["par"]).to(_dev())))
    sweep, _, _ = _posterior(case, p, plain, inverse=kind == "predict")
    if kind == "draws":        # the draws depend on the factor's ordering; the determinant does not
        return {"logdet": float(sweep(None)[0]), "x": None}
    hits = torch.zeros(T * ns, dtype=torch.float64, device=_dev())
    idx = torch.as_tensor(p["idx"]).to(_dev())
    hits[idx] = p["tau"]
    b = torch.zeros(T * ns, 1, dtype=torch.float64, device=_dev())
    b[idx, 0] = p["tau"] * torch.as_tensor(p["y"]).to(_dev())
    _, mu, Cd, _ = sweep(hits.reshape(T, ns), b.reshape(T, ns, 1))
    return {"mu": torch.cat(mu)[:, 0], "var": torch.cat([c.diagonal() for c in Cd])}
