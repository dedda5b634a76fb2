"""The solver's kernels on grids whose coefficient and weight arrays hold more than 2^31
entries: run on the CPU for the last nodes, with memory that is only mapped."""
import ctypes
import mmap

import numpy as np
import pytest

from host_kernels import compile_host, section

TAIL = r"""
struct Prod { int Mx, Ny, T, lead; Walk wk; const float *cf, *o32, *p; float *ap, *part; };
extern "C" void spmv_host(int Mx, int Ny, int T, int blk, const float* cf, const float* p, float* ap, float* part) {
  const int ng = (Mx * Ny * T + 31) / 32;
  Prod a = {Mx, Ny, T, 0, {1, ng, 1, ng, (ng + 7) / 8, (ng + 7) / 8}, cf, nullptr, p, ap, part};
  host::run({blk, 0, 0}, {(ng + 7) / 8, 1, 1}, 256, true, [](void* v) {
    Prod* a = static_cast<Prod*>(v);
    spmv32_kernel<1, 0>(a->Mx, a->Ny, a->T, 0.f, 0.f, 0.f, a->wk, 0, a->wk.ngroups, a->cf, a->o32, a->p, a->ap, a->part);
  }, &a);
}
struct App { int Mx, Ny, T; Walk wk; GWeights gw; const float* x; float *out, *part, *near; };
extern "C" void apply_host(int Mx, int Ny, int T, int blk, const float* w, const uint32_t* mask, const int* rank, int nob,
                           const uint32_t* near, const int* nrank, float* near_w, int ncap, const float* x, float* g,
                           float* gt, float* gt2, float* part) {
  const int Ns = Mx * Ny, ng = (Ns * T + 31) / 32;
  App a = {Mx, Ny, T, {1, ng, 1, ng, (ng + 7) / 8, (ng + 7) / 8},
           {w, mask, rank, nob, Ns, T, 1, near, nrank, near_w, ncap}, x, g, part, near_w};
  auto go = [&](void (*f)(void*)) { host::run({blk, 0, 0}, {(ng + 7) / 8, 1, 1}, 256, true, f, &a); };
  go([](void* v) { App* a = static_cast<App*>(v); near_rows_kernel(a->Mx, a->Ny, a->T, a->gw, a->near); });
  go([](void* v) {
    App* a = static_cast<App*>(v);
    g32_kernel<1, 0, 1>(a->Mx, a->Ny, a->T, a->wk, 0, a->wk.ngroups, a->gw, a->x, a->out, nullptr, nullptr);
  });
  a.out = gt;
  go([](void* v) {
    App* a = static_cast<App*>(v);
    g32_kernel<1, 1, 1>(a->Mx, a->Ny, a->T, a->wk, 0, a->wk.ngroups, a->gw, a->x, a->out, a->x, a->part);
  });
  a.out = gt2;
  a.gw.near = nullptr;  // every weight looked up
  go([](void* v) {
    App* a = static_cast<App*>(v);
    g32_kernel<1, 1, 2>(a->Mx, a->Ny, a->T, a->wk, 0, a->wk.ngroups, a->gw, a->x, a->out, a->x, a->part);
  });
}
"""


@pytest.fixture(scope="module")
def lib():
    parts = ["constexpr int kOff = 27;",
             section("pcg.cu", "template <int V>\nstruct alignas(4 * V) Cols", "// Fixed-order block sum"),
             section("pcg.cu", "struct Walk {", "// The same product for one column"),
             section("pcg.cu", "struct GWeights {", "// Bits of the nodes"),
             section("pcg.cu", "__device__ __forceinline__ int time_class", "// ------------------------------------------------------------ IC(0)")]
    return compile_host(parts, TAIL)


def _floats(count):
    """`count` floats of zeros, mapped but not held, after 2^31 more (where an index that wrapped would read)."""
    m = mmap.mmap(-1, 4 * (count + 2 ** 31), flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS | 0x4000)  # MAP_NORESERVE
    return np.frombuffer(m, np.float32)[2 ** 31:]


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _neighbours(k, Mx, Ny, T, r):
    t, c = divmod(k, Mx * Ny)
    y, x = divmod(c, Mx)
    for dt in (-1, 0, 1):
        for dy in range(-r, r + 1):
            for dx in range(-r, r + 1):
                if 0 <= x + dx < Mx and 0 <= y + dy < Ny and 0 <= t + dt < T:
                    yield dx, dy, dt, ((t + dt) * Ny + y + dy) * Mx + x + dx


# 27 nodes stays below 2^31 (larger grids are refused) while 69 or 81 cells do not
@pytest.mark.parametrize("Mx,Ny,T,step", [(40, 30, 1, 0), (5800, 5700, 1, 0), (5800, 5700, 2, 0), (5800, 5700, 2, 1)])
def test_product(lib, Mx, Ny, T, step):
    Ns, n = Mx * Ny, Mx * Ny * T
    assert 27 * n < 2 ** 31
    rng = np.random.default_rng(1)
    cf, p, ap = _floats(69 * Ns), _floats(n), _floats(n)
    part = np.zeros((n + 31) // 32 + 8, np.float32)
    blk = ((step + 1) * Ns - 4 * Mx) // 256 - 1  # a few rows before the end of the time step
    nodes = range(256 * blk, 256 * blk + 256)
    cells = np.array([k % Ns for k in nodes])
    cf.reshape(69, Ns)[:, cells] = rng.normal(size=(69, 256))
    for k in nodes:
        for _, _, _, q in _neighbours(k, Mx, Ny, T, 2):
            p[q] = 1 + q % 7
    lib.spmv_host(Mx, Ny, T, blk, _ptr(cf), _ptr(p), _ptr(ap), _ptr(part))
    for k in nodes:
        t, c = divmod(k, Ns)
        s = mag = 0.0
        for dx, dy, dt, q in _neighbours(k, Mx, Ny, T, 2):
            if dt == 0:
                v = float(cf[((0 if t == 0 and T > 1 else 25) + 5 * (dy + 2) + dx + 2) * Ns + c])
                if dx == dy == 0 and t < T - 1:
                    v += float(cf[68 * Ns + c])
            elif max(abs(dx), abs(dy)) <= 1:
                v = float(cf[((50 if dt > 0 else 59) + 3 * (dy + 1) + dx + 1) * Ns + c])
            else:
                continue
            s += v * float(p[q])
            mag += abs(v * float(p[q]))
        assert abs(ap[k] - s) <= 64 * 2.0 ** -24 * mag


@pytest.mark.parametrize("Mx,Ny,T", [(40, 30, 1), (5800, 5700, 1), (5800, 5700, 2)])
def test_preconditioner(lib, Mx, Ny, T):
    Ns, n = Mx * Ny, Mx * Ny * T
    rng = np.random.default_rng(2)
    blk = n // 256 - 1
    nodes = range(256 * blk, 256 * blk + 256)
    obs = np.array(nodes[40:200:23])
    nob, ncap = len(obs), 27 * len(obs)
    w, x, g, gt, gt2 = _floats(81 * Ns + 27 * nob), *[_floats(n) for _ in range(4)]
    ring = sorted({q for k in nodes for _, _, _, q in _neighbours(k, Mx, Ny, T, 1)})
    cls = lambda t: 0 if t == 0 else (2 if t == T - 1 else 1)
    for k in ring:
        x[k] = rng.normal()
        t, c = divmod(k, Ns)
        w[(27 * cls(t) + np.arange(27)) * Ns + c] = rng.normal(size=27)
    w[81 * Ns:] = rng.normal(size=27 * nob)
    mask, near = np.zeros((n + 31) // 32, np.uint32), np.zeros((n + 31) // 32, np.uint32)
    for a, bits in ((obs, mask), ({q for k in obs for _, _, _, q in _neighbours(k, Mx, Ny, T, 1)}, near)):
        for k in a:
            bits[k >> 5] |= np.uint32(1 << (k & 31))
    def ranks(bits):
        c = np.zeros(len(bits), np.int64)
        for i in np.flatnonzero(bits):
            c[i] = bin(int(bits[i])).count("1")
        return (np.cumsum(c) - c).astype(np.int32)
    rank, nrank = ranks(mask), ranks(near)
    near_w = np.zeros(27 * ncap, np.float32)
    part = np.zeros((n + 31) // 32 + 8, np.float32)
    lib.apply_host(Mx, Ny, T, blk, _ptr(w), _ptr(mask), _ptr(rank), nob, _ptr(near), _ptr(nrank), _ptr(near_w), ncap,
                   _ptr(x), _ptr(g), _ptr(gt), _ptr(gt2), _ptr(part))
    assert np.array_equal(gt[nodes[0]:nodes[-1] + 1], gt2[nodes[0]:nodes[-1] + 1])
    row = {int(k): j for j, k in enumerate(obs)}
    def weight(k, o):
        if k in row:
            return float(w[81 * Ns + o * nob + row[k]])
        t, c = divmod(k, Ns)
        return float(w[(27 * cls(t) + o) * Ns + c])
    for k in nodes:
        s = st = mag = 0.0
        for dx, dy, dt, q in _neighbours(k, Mx, Ny, T, 1):
            o = 9 * (dt + 1) + 3 * (dy + 1) + dx + 1
            a, b = weight(k, o) * float(x[q]), weight(q, 26 - o) * float(x[q])
            s, st, mag = s + a, st + b, mag + abs(a) + abs(b)
        assert abs(g[k] - s) <= 64 * 2.0 ** -24 * mag and abs(gt[k] - st) <= 64 * 2.0 ** -24 * mag
