// Learned space-time preconditioner and preconditioned conjugate gradients for
// A = Q (+ tau S^T S) on grids too large to factor.
//
// The preconditioner is a factorised sparse approximate inverse M^-1 = G^T G.
// G is a 27-point stencil on the (x, y, t) lattice (dx, dy, dt in {-1, 0, 1})
// whose per-node weights come from a small network that reads the node's own
// row of A: w_o(p) = (delta_o,centre + N(f_p)_o) / sqrt(A_pp), with
// f_p = A_p,. / A_pp over the 43-slot stencil (centre dropped) and N a
// 42-32-32-27 perceptron with tanh activations.  A zero last layer gives the
// Jacobi preconditioner.  Training minimises
//   L = E_z || z - G A G^T z ||^2 / (n k)
// over probe blocks z (n x k), i.e. drives G A G^T towards the identity; the
// gradient with respect to the weights is
//   dL/dw_o(p) = -2/(n k) sum_r (e_pr u_(p+o)r + z_pr g_(p+o)r)
// with y = G^T z, u = A y, e = z - G u, g = A G^T e, and flows into the network
// through its own backward kernel.  Parameters live in caller-owned FP32
// device memory; every reduction is a fixed-order two-pass sum, so results are
// deterministic.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <vector>

#include "engine.cuh"

namespace spde {

namespace {

constexpr int kFeat = kPcFeat, kHid = kPcHidden, kOff = kPcOffsets;
constexpr int kW1 = 0, kB1 = kW1 + kHid * kFeat, kW2 = kB1 + kHid, kB2 = kW2 + kHid * kHid, kW3 = kB2 + kHid,
              kB3 = kW3 + kOff * kHid, kNP = kB3 + kOff;
static_assert(kNP == kPcParams, "parameter layout");
constexpr int kAct = kFeat + 2 * kHid + 1;  // per node: f, h1, h2, 1 / sqrt(A_pp)
constexpr int kCentre43 = 21;               // centre slot of the 43-slot layout

__device__ __forceinline__ void off27(int o, int* dx, int* dy, int* dt) {
  *dt = o / 9 - 1;
  *dy = (o / 3) % 3 - 1;
  *dx = o % 3 - 1;
}

// 43-slot layout offsets (dt = -1: 3 x 3, dt = 0: 5 x 5, dt = +1: 3 x 3)
__device__ __forceinline__ void off43(int s, int* dx, int* dy, int* dt) {
  if (s < 9) { *dt = -1; *dy = s / 3 - 1; *dx = s % 3 - 1; }
  else if (s < 34) { *dt = 0; *dy = (s - 9) / 5 - 2; *dx = (s - 9) % 5 - 2; }
  else { *dt = 1; *dy = (s - 34) / 3 - 1; *dx = (s - 34) % 3 - 1; }
}

__device__ __forceinline__ bool inside(const QStencil& q, int x, int y, int t) {
  return x >= 0 && x < q.Mx && y >= 0 && y < q.Ny && t >= 0 && t < q.T;
}

// Features, network forward and the 27 G weights of the row of A at (cell c,
// time t), whose diagonal carries the observation term `obs_term`; `act`
// (optional) receives the activations a gradient step needs.
__device__ __forceinline__ void pc_network(const QStencil& q, int c, int t, double obs_term, const float* sp,
                                           float* wout, float* act) {
  const int y = c / q.Mx, x = c - y * q.Mx;
  double diag = qval(q, c, t, 0, 0, 0) + obs_term;
  if (!(diag > 0.0)) diag = 1.0;
  const double rd = 1.0 / diag;
  float f[kFeat];
#pragma unroll
  for (int s = 0; s < 43; ++s) {
    if (s == kCentre43) continue;
    int dx, dy, dt;
    off43(s, &dx, &dy, &dt);
    double v = 0.0;
    if ((q.T > 1 || dt == 0) && inside(q, x + dx, y + dy, t + dt)) v = qval(q, c, t, dx, dy, dt) * rd;
    f[s < kCentre43 ? s : s - 1] = float(v);
  }
  float h1[kHid], h2[kHid];
#pragma unroll 4
  for (int i = 0; i < kHid; ++i) {
    float a = sp[kB1 + i];
#pragma unroll
    for (int j = 0; j < kFeat; ++j) a = fmaf(sp[kW1 + i * kFeat + j], f[j], a);
    h1[i] = tanhf(a);
  }
#pragma unroll 4
  for (int i = 0; i < kHid; ++i) {
    float a = sp[kB2 + i];
#pragma unroll
    for (int j = 0; j < kHid; ++j) a = fmaf(sp[kW2 + i * kHid + j], h1[j], a);
    h2[i] = tanhf(a);
  }
  const float s = float(rsqrt(diag));
  for (int o = 0; o < kOff; ++o) {
    float a = sp[kB3 + o];
#pragma unroll
    for (int j = 0; j < kHid; ++j) a = fmaf(sp[kW3 + o * kHid + j], h2[j], a);
    int dx, dy, dt;
    off27(o, &dx, &dy, &dt);
    const bool in = inside(q, x + dx, y + dy, t + dt);
    wout[o] = in ? ((o == 13 ? 1.f : 0.f) + a) * s : 0.f;
  }
  if (act) {
#pragma unroll
    for (int j = 0; j < kFeat; ++j) act[j] = f[j];
#pragma unroll
    for (int j = 0; j < kHid; ++j) act[kFeat + j] = h1[j];
#pragma unroll
    for (int j = 0; j < kHid; ++j) act[kFeat + kHid + j] = h2[j];
    act[kAct - 1] = s;
  }
}

// G weights of every node, offset-major (w[o n + p]), one thread per node.
// The activations of a block's nodes are contiguous: staged in shared memory and
// written in order.
__global__ void __launch_bounds__(128) pc_forward_kernel(QStencil q, const double* __restrict__ obs, double tau,
                                                         const float* __restrict__ prm, float* __restrict__ w,
                                                         float* __restrict__ act) {
  extern __shared__ float fsm[];
  float* sp = fsm;
  float* sact = fsm + kNP;  // 128 x kAct (with act)
  for (int i = threadIdx.x; i < kNP; i += blockDim.x) sp[i] = prm[i];
  __syncthreads();
  const int64_t n = int64_t(q.Ns) * q.T;
  const int64_t p0 = int64_t(blockIdx.x) * 128, p = p0 + threadIdx.x;
  if (p < n) {
    const int t = int(p / q.Ns), c = int(p - int64_t(t) * q.Ns);
    float wo[kOff];
    pc_network(q, c, t, obs ? tau * obs[p] : 0.0, sp, wo, act ? sact + threadIdx.x * kAct : nullptr);
#pragma unroll
    for (int o = 0; o < kOff; ++o) w[int64_t(o) * n + p] = wo[o];
  }
  if (act) {
    __syncthreads();
    const int cnt = int(n - p0 < 128 ? n - p0 : 128) * kAct;
    for (int i = threadIdx.x; i < cnt; i += 128) act[p0 * kAct + i] = sact[i];
  }
}

// Compact weights.  A node's row of A depends on its time only through three
// classes (first step, interior steps, last step: the stencil coefficients are
// time-invariant) unless the node is observed, so G has one row per (class,
// cell) and one per distinct observed node: w[(k 27 + o) Ns + c] for class k,
// then w[27 3 Ns + o nob + j] for the j-th observed node.  One thread per row.
__global__ void __launch_bounds__(128) pc_forward_compact_kernel(QStencil q, const double* __restrict__ obs,
                                                                 double tau, const int* __restrict__ obs_nodes,
                                                                 int nob, const float* __restrict__ prm,
                                                                 float* __restrict__ w) {
  __shared__ float sp[kNP];
  for (int i = threadIdx.x; i < kNP; i += blockDim.x) sp[i] = prm[i];
  __syncthreads();
  const int64_t ncls = int64_t(3) * q.Ns;
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= ncls + nob) return;
  float wo[kOff];
  if (e < ncls) {
    const int k = int(e / q.Ns), c = int(e - int64_t(k) * q.Ns);
    const int t = k == 0 ? 0 : (k == 1 ? (q.T > 2 ? 1 : 0) : q.T - 1);
    pc_network(q, c, t, 0.0, sp, wo, nullptr);
#pragma unroll
    for (int o = 0; o < kOff; ++o) w[(int64_t(k) * kOff + o) * q.Ns + c] = wo[o];
  } else {
    const int j = int(e - ncls);
    const int p = obs_nodes[j];
    const int t = p / q.Ns, c = p - t * q.Ns;
    pc_network(q, c, t, obs ? tau * obs[p] : 0.0, sp, wo, nullptr);
#pragma unroll
    for (int o = 0; o < kOff; ++o) w[ncls * kOff + int64_t(o) * nob + j] = wo[o];
  }
}

// out = G x (transpose = 0) or G^T x (transpose = 1); x, out n x nrhs row-major;
// weights offset-major (w[o n + p]), so every offset's read is coalesced.  The
// 27 offsets are unrolled (compile-time displacements, loads issued together);
// node indices fit in 32 bits (checked by the caller).
template <int TRANS, typename TIn, typename TOut>
__global__ void pc_apply_kernel(QStencil q, const float* __restrict__ w, const TIn* __restrict__ x,
                                TOut* __restrict__ out, int nrhs) {
  const int n = q.Ns * q.T;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n * nrhs) return;
  const int p = nrhs == 1 ? e : e / nrhs;
  const int r = e - p * nrhs;
  const int t = p / q.Ns, c = p - t * q.Ns;
  const int y = c / q.Mx, xx = c - y * q.Mx;
  const int sy = q.Mx, st = q.Ns;
  // FP32 arithmetic: a preconditioner only has to be a fixed SPD operator, and
  // FP64 is a narrow pipe on this part
  float acc = 0.f;
#pragma unroll
  for (int o = 0; o < kOff; ++o) {
    const int dx = o % 3 - 1, dy = (o / 3) % 3 - 1, dt = o / 9 - 1;
    const int sgn = TRANS ? -1 : 1;
    const int x2 = xx + sgn * dx, y2 = y + sgn * dy, t2 = t + sgn * dt;
    if (x2 < 0 || x2 >= q.Mx || y2 < 0 || y2 >= q.Ny || t2 < 0 || t2 >= q.T) continue;
    const int nb = p + sgn * (dt * st + dy * sy + dx);
    const float wv = TRANS ? w[int64_t(o) * n + nb] : w[int64_t(o) * n + p];
    acc = fmaf(wv, float(x[int64_t(nb) * nrhs + r]), acc);
  }
  out[e] = TOut(acc);
}

__global__ void pc_sub_kernel(const double* __restrict__ z, double* __restrict__ v, int64_t len) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < len) v[i] = z[i] - v[i];
}

// dL/d(network output) per node: (sum_r e_pr u_(p+o)r + z_pr g_(p+o)r) * scale * s_p.
// NR columns (0: nrhs of them) with the node's own values held in registers.
template <int NR>
__global__ void __launch_bounds__(128) pc_wgrad_kernel(QStencil q, const double* __restrict__ z,
                                                       const double* __restrict__ e, const double* __restrict__ u,
                                                       const double* __restrict__ g, int nrhs, double scale,
                                                       const float* __restrict__ act, float* __restrict__ dout) {
  __shared__ float so[128 * kOff];
  const int64_t n = int64_t(q.Ns) * q.T;
  const int64_t p0 = int64_t(blockIdx.x) * 128, p = p0 + threadIdx.x;
  if (p < n) {
    const int t = int(p / q.Ns), c = int(p - int64_t(t) * q.Ns);
    const int y = c / q.Mx, x = c - y * q.Mx;
    const double s = act[p * kAct + kAct - 1];
    double ep[NR > 0 ? NR : 1], zp[NR > 0 ? NR : 1];
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      ep[r] = e[p * NR + r];
      zp[r] = z[p * NR + r];
    }
#pragma unroll 3
    for (int o = 0; o < kOff; ++o) {
      int dx, dy, dt;
      off27(o, &dx, &dy, &dt);
      double acc = 0.0;
      if (inside(q, x + dx, y + dy, t + dt)) {
        const int64_t nb = p + (int64_t(dt) * q.Ny + dy) * q.Mx + dx;
        if (NR > 0) {
#pragma unroll
          for (int r = 0; r < NR; ++r) {
            acc = fma(ep[r], u[nb * NR + r], acc);
            acc = fma(zp[r], g[nb * NR + r], acc);
          }
        } else {
          for (int r = 0; r < nrhs; ++r) {
            acc = fma(e[p * nrhs + r], u[nb * nrhs + r], acc);
            acc = fma(z[p * nrhs + r], g[nb * nrhs + r], acc);
          }
        }
      }
      so[threadIdx.x * kOff + o] = float(acc * scale * s);
    }
  }
  __syncthreads();
  const int cnt = int(n - p0 < 128 ? n - p0 : 128) * kOff;  // the block's rows are contiguous
  for (int i = threadIdx.x; i < cnt; i += 128) dout[p0 * kOff + i] = so[i];
}

// Network backward: per block of kBwNodes nodes, the parameter gradient of the
// block's nodes into its own row of `part` (nblocks x kNP).
// Bound: shared-memory reads; every product is tiled in registers.
constexpr int kBwNodes = 64;
constexpr int kBwThreads = 192;
static_assert(kFeat == 42 && kHid == 32 && kOff == 27, "tiles of the weight gradients");
// out[i ldo + j] = sum over nodes a of D[a ldd + i] H[a ldh + j], R x C entries
template <int R, int C>
__device__ __forceinline__ void weight_tile(const float* D, int ldd, const float* H, int ldh, float* out, int ldo) {
  float acc[R][C];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < C; ++j) acc[i][j] = 0.f;
#pragma unroll 4
  for (int a = 0; a < kBwNodes; ++a) {
    float d[R], h[C];
#pragma unroll
    for (int i = 0; i < R; ++i) d[i] = D[a * ldd + i];
#pragma unroll
    for (int j = 0; j < C; ++j) h[j] = H[a * ldh + j];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < C; ++j) acc[i][j] = fmaf(d[i], h[j], acc[i][j]);
  }
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < C; ++j) out[i * ldo + j] = acc[i][j];
}
__global__ void __launch_bounds__(kBwThreads) pc_backward_kernel(int64_t n, const float* __restrict__ prm,
                                                          const float* __restrict__ act,
                                                          const float* __restrict__ dout, float* __restrict__ part) {
  extern __shared__ float sm[];
  float* sW2 = sm;                              // kHid * kHid
  float* sW3 = sW2 + kHid * kHid;               // kOff * kHid
  float* sf = sW3 + kOff * kHid;                // kBwNodes * kFeat
  float* sh1 = sf + kBwNodes * kFeat;           // kBwNodes * kHid
  float* sh2 = sh1 + kBwNodes * kHid;
  float* sdo = sh2 + kBwNodes * kHid;           // kBwNodes * kOff
  float* sd2 = sdo + kBwNodes * kOff;           // kBwNodes * kHid
  float* sd1 = sd2 + kBwNodes * kHid;
  const int tid = threadIdx.x;
  for (int i = tid; i < kHid * kHid; i += blockDim.x) sW2[i] = prm[kW2 + i];
  for (int i = tid; i < kOff * kHid; i += blockDim.x) sW3[i] = prm[kW3 + i];
  const int64_t p0 = int64_t(blockIdx.x) * kBwNodes;
  const int cnt = n - p0 < kBwNodes ? int(n - p0) : kBwNodes;
  for (int i = tid; i < kBwNodes * kFeat; i += blockDim.x) {
    const int a = i / kFeat, j = i - a * kFeat;
    sf[i] = a < cnt ? act[(p0 + a) * kAct + j] : 0.f;
  }
  for (int i = tid; i < kBwNodes * kHid; i += blockDim.x) {
    const int a = i / kHid, j = i - a * kHid;
    sh1[i] = a < cnt ? act[(p0 + a) * kAct + kFeat + j] : 0.f;
    sh2[i] = a < cnt ? act[(p0 + a) * kAct + kFeat + kHid + j] : 0.f;
  }
  for (int i = tid; i < kBwNodes * kOff; i += blockDim.x) {
    const int a = i / kOff;
    sdo[i] = a < cnt ? dout[(p0 + a) * kOff + (i - a * kOff)] : 0.f;
  }
  __syncthreads();
  // dh2 = W3^T dout (1 - h2^2), then dh1 = W2^T dh2 (1 - h1^2): lane = hidden unit,
  // eight nodes per thread
  const int j = tid & 31;
  for (int a0 = 8 * (tid >> 5); a0 < kBwNodes; a0 += 8 * (kBwThreads / 32)) {
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
#pragma unroll 3
    for (int o = 0; o < kOff; ++o) {
      const float w = sW3[o * kHid + j];
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = fmaf(w, sdo[(a0 + i) * kOff + o], acc[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float h = sh2[(a0 + i) * kHid + j];
      sd2[(a0 + i) * kHid + j] = acc[i] * (1.f - h * h);
    }
  }
  __syncthreads();
  for (int a0 = 8 * (tid >> 5); a0 < kBwNodes; a0 += 8 * (kBwThreads / 32)) {
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
#pragma unroll 4
    for (int k = 0; k < kHid; ++k) {
      const float w = sW2[k * kHid + j];
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = fmaf(w, sd2[(a0 + i) * kHid + k], acc[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float h = sh1[(a0 + i) * kHid + j];
      sd1[(a0 + i) * kHid + j] = acc[i] * (1.f - h * h);
    }
  }
  __syncthreads();
  // dW = D^T H over the block's nodes, one register tile per thread: 56 tiles of
  // 4 x 6 for W1, 64 of 4 x 4 for W2, 72 of 3 x 4 for W3
  float* out = part + int64_t(blockIdx.x) * kNP;
  if (tid < 56)
    weight_tile<4, 6>(sd1 + 4 * (tid / 7), kHid, sf + 6 * (tid % 7), kFeat, out + kW1 + 4 * (tid / 7) * kFeat + 6 * (tid % 7),
                      kFeat);
  else if (tid < 120)
    weight_tile<4, 4>(sd2 + 4 * ((tid - 56) / 8), kHid, sh1 + 4 * ((tid - 56) % 8), kHid,
                      out + kW2 + 4 * ((tid - 56) / 8) * kHid + 4 * ((tid - 56) % 8), kHid);
  else
    weight_tile<3, 4>(sdo + 3 * ((tid - 120) / 8), kOff, sh2 + 4 * ((tid - 120) % 8), kHid,
                      out + kW3 + 3 * ((tid - 120) / 8) * kHid + 4 * ((tid - 120) % 8), kHid);
  if (tid < kHid + kHid + kOff) {  // biases
    const float* d = tid < kHid ? sd1 + tid : tid < 2 * kHid ? sd2 + tid - kHid : sdo + tid - 2 * kHid;
    const int ld = tid < 2 * kHid ? kHid : kOff;
    float acc = 0.f;
    for (int a = 0; a < kBwNodes; ++a) acc += d[a * ld];
    out[tid < kHid ? kB1 + tid : tid < 2 * kHid ? kB2 + tid - kHid : kB3 + tid - 2 * kHid] = acc;
  }
}

// grad[e] = sum over blocks of part[b][e] in FP64 and a fixed order: kColParts CTAs
// share the blocks of every 128 columns, the last of them to finish adds their sums
constexpr int kColParts = 32;
__global__ void __launch_bounds__(128) pc_colsum_kernel(const float* __restrict__ part, int nb,
                                                        double* __restrict__ sums, unsigned* __restrict__ arrived,
                                                        float* __restrict__ grad) {
  __shared__ bool last;
  const int e = blockIdx.x * 128 + threadIdx.x;
  const int per = (nb + kColParts - 1) / kColParts, b0 = int(blockIdx.y) * per, b1 = min(nb, b0 + per);
  double acc = 0.0;
  if (e < kNP) {
#pragma unroll 8
    for (int b = b0; b < b1; ++b) acc += part[int64_t(b) * kNP + e];
    sums[int64_t(blockIdx.y) * kNP + e] = acc;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&arrived[blockIdx.x], 1u) == kColParts - 1;
  __syncthreads();
  if (!last || e >= kNP) return;
  __threadfence();
  acc = 0.0;
#pragma unroll 8
  for (int b = 0; b < kColParts; ++b) acc += __ldcg(sums + int64_t(b) * kNP + e);
  grad[e] = float(acc);
}

// Column-wise dot products of a and b (n x nrhs row-major): two-pass, fixed order.
constexpr int kDotBlocks = 256;
__global__ void pc_dot_partial_kernel(const double* __restrict__ a, const double* __restrict__ b, int64_t n, int nrhs,
                                      double* __restrict__ part) {
  __shared__ double red[256];
  for (int r = 0; r < nrhs; ++r) {
    double acc = 0.0;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
      acc += a[i * nrhs + r] * b[i * nrhs + r];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int k = 128; k > 0; k >>= 1) {
      if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
      __syncthreads();
    }
    if (threadIdx.x == 0) part[int64_t(r) * gridDim.x + blockIdx.x] = red[0];
    __syncthreads();
  }
}
// The same for many columns: lane = column within a 32-column chunk
// (blockIdx.y), warps stride over the rows, so each row segment is read
// contiguously; part[r * gridDim.x + block] as in pc_dot_partial_kernel.
__global__ void pc_dot_wide_kernel(const double* __restrict__ a, const double* __restrict__ b, int64_t n, int nrhs,
                                   double* __restrict__ part) {
  __shared__ double red[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = blockIdx.y * 32 + lane;
  double acc = 0.0;
  if (r < nrhs)
    for (int64_t i = int64_t(blockIdx.x) * 8 + warp; i < n; i += int64_t(gridDim.x) * 8)
      acc += a[i * nrhs + r] * b[i * nrhs + r];
  red[warp][lane] = acc;
  __syncthreads();
  if (warp == 0 && r < nrhs) {
    double s = 0.0;
    for (int w = 0; w < 8; ++w) s += red[w][lane];
    part[int64_t(r) * gridDim.x + blockIdx.x] = s;
  }
}

__global__ void pc_dot_final_kernel(const double* __restrict__ part, int nblocks, int nrhs, double* __restrict__ out) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nrhs) return;
  double acc = 0.0;
  for (int b = 0; b < nblocks; ++b) acc += part[int64_t(r) * nblocks + b];
  out[r] = acc;
}

// z -= omega D^-1 (A z) for one damped-Jacobi sweep (az = A z)
__global__ void jacobi_sweep_kernel(QStencil q, const double* __restrict__ obs, double tau, double omega,
                                    const double* __restrict__ az, double* __restrict__ z, int nrhs) {
  const int64_t n = int64_t(q.Ns) * q.T;
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= n * nrhs) return;
  const int64_t p = e / nrhs;
  const int t = int(p / q.Ns), c = int(p - int64_t(t) * q.Ns);
  const double d = qval(q, c, t, 0, 0, 0) + (obs ? tau * obs[p] : 0.0);
  z[e] -= omega * az[e] / d;
}
// wd = omega / diag(A) per node
__global__ void jacobi_weight_kernel(QStencil q, const double* __restrict__ obs, double tau, double omega,
                                     double* __restrict__ wd) {
  const int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (p >= int64_t(q.Ns) * q.T) return;
  const int t = int(p / q.Ns), c = int(p - int64_t(t) * q.Ns);
  wd[p] = omega / (qval(q, c, t, 0, 0, 0) + (obs ? tau * obs[p] : 0.0));
}
// z[:, r] *= 1 / sqrt(ss[r] / n)
__global__ void col_scale_kernel(double* __restrict__ z, const double* __restrict__ ss, int64_t n, int nrhs) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= n * nrhs) return;
  const int r = int(e % nrhs);
  const double ms = ss[r] / double(n);
  if (ms > 0.0) z[e] *= 1.0 / sqrt(ms);
}

__global__ void adam_kernel(float* __restrict__ prm, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, int n, float lr, float b1, float b2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  prm[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

inline int nblk(int64_t n, int b = 256) { return int((n + b - 1) / b); }

double* scratch(Plan* p, size_t elems) {
  if (elems > p->pc_cap) {
    cudaFree(p->d_pc);
    p->d_pc = nullptr;
    p->pc_cap = 0;
    if (cudaMalloc(&p->d_pc, elems * sizeof(double)) != cudaSuccess) return nullptr;
    p->pc_cap = elems;
  }
  return static_cast<double*>(p->d_pc);
}

void col_dots(Plan* p, const double* a, const double* b, int nrhs, double* part, double* out) {
  if (nrhs == 1) {
    pc_dot_partial_kernel<<<kDotBlocks, 256, 0, p->stream>>>(a, b, p->sym.n, 1, part);
  } else {
    const dim3 grid(kDotBlocks, (nrhs + 31) / 32);
    pc_dot_wide_kernel<<<grid, 256, 0, p->stream>>>(a, b, p->sym.n, nrhs, part);
  }
  pc_dot_final_kernel<<<nblk(nrhs, 64), 64, 0, p->stream>>>(part, kDotBlocks, nrhs, out);
}

// Square root of Q: Q = B^T B with B (n x n) stacking, for the initial field,
// V^-1/2 A0 (rows (c, 0)) and, for each step t -> t + 1, sqrt(c qs_c) (A x_(t+1)
// / V - x_t) (rows (c, t + 1)); for a spatial model (T = 1) B = V^-1/2 A.  A and
// A0 are the 9-point implicit-Euler and initial-field operators (A_geo[c 9 + p]
// = A[c, c + off_p], off_p = (p % 3 - 1, p / 3 - 1)), qs = V kappa^2, c =
// 1 / (dt sigma) (spdes/advection_diffusion2D.py:101-116 written as a sum of squares).
// out = B x (TRANS = 0) or B^T x (TRANS = 1), n x nrhs row-major.
template <int TRANS>
__global__ void qsqrt_kernel(int Mx, int Ny, int T, const double* __restrict__ Ag, const double* __restrict__ A0g,
                             const double* __restrict__ qs, double V, double cfac, const double* __restrict__ x,
                             double* __restrict__ out, int nrhs) {
  const int Ns = Mx * Ny, n = Ns * T;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n * nrhs) return;
  const int k = nrhs == 1 ? e : e / nrhs;
  const int r = e - k * nrhs;
  const int t = k / Ns, c = k - t * Ns;
  const int cy = c / Mx, cx = c - cy * Mx;
  const double rv = 1.0 / sqrt(V);
  double acc = 0.0;
  if (!TRANS) {
    // row (c, t)
    const double* Ar = (T > 1 && t == 0 ? A0g : Ag) + int64_t(c) * 9;
    double sum = 0.0;
#pragma unroll
    for (int p = 0; p < 9; ++p) {
      const int x2 = cx + p % 3 - 1, y2 = cy + p / 3 - 1;
      if (x2 < 0 || x2 >= Mx || y2 < 0 || y2 >= Ny) continue;
      sum = fma(Ar[p], x[int64_t(t * Ns + y2 * Mx + x2) * nrhs + r], sum);
    }
    if (T == 1 || t == 0) acc = rv * sum;
    else acc = sqrt(cfac * qs[c]) * (sum / V - x[int64_t((t - 1) * Ns + c) * nrhs + r]);
  } else {
    // column (c, t): rows (c', t) with c = c' + off_p, and the -1 of row (c, t + 1)
#pragma unroll
    for (int p = 0; p < 9; ++p) {
      const int x2 = cx - (p % 3 - 1), y2 = cy - (p / 3 - 1);
      if (x2 < 0 || x2 >= Mx || y2 < 0 || y2 >= Ny) continue;
      const int c2 = y2 * Mx + x2;
      const double xe = x[int64_t(t * Ns + c2) * nrhs + r];
      if (T == 1 || t == 0) acc = fma(rv * (T > 1 ? A0g : Ag)[int64_t(c2) * 9 + p], xe, acc);
      else acc = fma(sqrt(cfac * qs[c2]) * Ag[int64_t(c2) * 9 + p] / V, xe, acc);
    }
    if (T > 1 && t + 1 < T) acc -= sqrt(cfac * qs[c]) * x[int64_t((t + 1) * Ns + c) * nrhs + r];
  }
  out[e] = acc;
}

// ------------------------------------------------------------ FP32 PCG
// The iteration runs in FP32 (stencil product, vectors, preconditioner): FP64
// is a narrow pipe on this part, and an FP64 stencil product is bound by it.
// The solution is accumulated and the residual recomputed in FP64 whenever
// the recursive FP32 residual has fallen by kReplaceDrop (reliable updates),
// so the reported tolerance is always met by the true FP64 residual.
// Inside the solver every vector is stored column by column (column r of an
// FP32 vector at v + r n), and each kernel takes its column from blockIdx.y or
// blockIdx.z.

// FP32 copies of the stencil coefficients, slot-major (cf[s Ns + c]): slots
// 0-24 first diagonal block (T > 1), 25-49 interior diagonal block, 50-58 the
// block to t + 1, 59-67 the neighbours' blocks to t - 1 mirrored onto this
// cell, 68 c Qs.
constexpr int kCoef32 = 69;
__global__ void coef32_kernel(QStencil q, float* __restrict__ cf) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= q.Ns) return;
  const int cy = c / q.Mx, cx = c - cy * q.Mx;
  const int64_t Ns = q.Ns;
  const bool st = q.T > 1 && !q.sep;
  for (int s = 0; s < 25; ++s) {
    cf[s * Ns + c] = st ? float(q.Q0[int64_t(c) * 25 + s]) : 0.f;
    cf[(25 + s) * Ns + c] = float(q.QA[int64_t(c) * 25 + s]);
  }
  for (int s = 0; s < 9; ++s) {
    const int dx = s % 3 - 1, dy = s / 3 - 1;
    const bool in = cx + dx >= 0 && cx + dx < q.Mx && cy + dy >= 0 && cy + dy < q.Ny;
    cf[(50 + s) * Ns + c] = st ? float(q.QO[int64_t(c) * 9 + s]) : 0.f;
    cf[(59 + s) * Ns + c] = (st && in) ? float(q.QO[int64_t(c + dy * q.Mx + dx) * 9 + (8 - s)]) : 0.f;
  }
  cf[68 * Ns + c] = st ? float(q.cQs[c]) : 0.f;
}

// obs32[k] = tau obs[k] in FP32 (the observation term of the diagonal)
__global__ void obs32_kernel(const double* __restrict__ obs, double tau, float* __restrict__ o32, int64_t n) {
  const int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k < n) o32[k] = float(tau * obs[k]);
}

// FP32 vectors of the solver hold their columns in groups of four (four values per
// node side by side, one 16-byte access), then a group of two and single
// columns; `packed` false keeps every column by itself (IC(0)).  Column c of
// node k lies at lead n + width k + (c - lead) for the group [lead, lead + width).
struct ColGroup {
  int lead, width;
};
__host__ __device__ __forceinline__ ColGroup col_group(int c, int nrhs, int packed) {
  if (!packed) return {c, 1};
  const int n4 = nrhs & ~3;
  if (c < n4) return {c & ~3, 4};
  if ((nrhs & 2) && c < n4 + 2) return {n4, 2};
  return {c, 1};
}
__device__ __forceinline__ int64_t col_elem(int c, int64_t k, int64_t n, int nrhs, int packed) {
  const ColGroup g = col_group(c, nrhs, packed);
  return g.lead * n + g.width * k + (c - g.lead);
}

// row-major FP64 (n x nrhs) -> grouped FP32, and x += xc back (xc = 0)
__global__ void to32cm_kernel(const double* __restrict__ v, float* __restrict__ o, int64_t n, int nrhs, int packed) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= n * nrhs) return;
  const int64_t k = e / nrhs;
  o[col_elem(int(e - k * nrhs), k, n, nrhs, packed)] = float(v[e]);
}
__global__ void acc64cm_kernel(double* __restrict__ x, float* __restrict__ xc, int64_t n, int nrhs, int packed) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= n * nrhs) return;
  const int64_t k = e / nrhs;
  const int64_t f = col_elem(int(e - k * nrhs), k, n, nrhs, packed);
  x[e] += double(xc[f]);
  xc[f] = 0.f;
}

// V values of one node (V = 1, 2 or 4 columns of a group)
template <int V>
struct alignas(4 * V) Cols {
  float v[V];
};

// Fixed-order block sum of one float per thread into part[] (thread 0 writes)
__device__ __forceinline__ double block_sum(float v, float* red) {
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < int(blockDim.x >> 5); ++w) s += red[w];
  return s;
}

// The per-node kernels (stencil product, G, G^T) work on 32-node warps: warp group g
// holds the nodes 32 g .. 32 g + 31 in node order, and the partial sums of the dot
// products are those of a group (summed eight at a time by the scalar kernel).
// A CTA's eight warps take groups R = round(Mx / 32) apart, i.e. nearly the same
// columns of eight consecutive grid rows, and walk `steps` time steps with them in
// strides of P = round(Ns / 32) groups, at most 16 nodes off the same cells: the
// neighbours' vector values and the cells' coefficients (or rows of G) that a step
// needs are then mostly in L1, from another warp or from the step before.
struct Walk {
  int R, P, steps, ngroups;  // groups per grid row and per time step, steps per CTA, groups in all
  int rows8, bx;             // eight-row tiles and CTAs per time step
};
__device__ __forceinline__ int walk_group(const Walk& wk, int j) {
  const int by = int(blockIdx.x) / wk.bx, cta = int(blockIdx.x) - by * wk.bx;
  const int ry = cta / wk.R;
  const int a1 = 8 * ry + int(threadIdx.x >> 5), a = (cta - ry * wk.R) + wk.R * a1;
  const int64_t g = a + int64_t(by * wk.steps + j) * wk.P;
  return a < wk.P && g < wk.ngroups ? int(g) : -1;
}
__device__ __forceinline__ float warp_sum(float v) {
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}

// ap = A p in FP32 for the columns [lead + V y, + V), one thread per node and V
// columns, and the warp groups' sums of p . ap into part[col gpad + group].  Node
// offsets fit in 32 bits (27 n < 2^31, checked by the caller), coefficient offsets in 32 bits
// without sign: below 50 Ns with one time step, below 69 Ns with two or more.
// Bound: L1 / L2 loads (43 coefficients and 43 V vector values per node).  Four
// columns per thread share the coefficients' loads and the index arithmetic.
// Measured at 200 x 200 x 24: 16 columns 155 us (417 with one column per thread), at
// 400 x 400 x 48 one column 178 us (228); with a branch per neighbour instead of
// a zero coefficient 356 us for the 16 columns.  Long runs of steps of one column go
// to spmv32_steps_kernel below; with four columns its registers leave too few warps
// (171 us against 155).
template <int V, int SEP>
__global__ void __launch_bounds__(256, 4) spmv32_kernel(int Mx, int Ny, int T, float qe, float qm, float qo,
                                                        Walk wk, int lead, int gpad, const float* __restrict__ cf,
                                                        const float* __restrict__ o32, const float* __restrict__ pv,
                                                        float* __restrict__ apv, float* __restrict__ part) {
  const int Ns = Mx * Ny, n = Ns * T, lane = threadIdx.x & 31;
  const int c0 = lead + V * int(blockIdx.y);
  const Cols<V>* x = reinterpret_cast<const Cols<V>*>(pv + int64_t(c0) * n);
  Cols<V>* out = reinterpret_cast<Cols<V>*>(apv + int64_t(c0) * n);
  for (int j = 0; j < wk.steps; ++j) {
    const int g = walk_group(wk, j);
    if (g < 0) continue;
    const int k = 32 * g + lane;
    float dot[V];
#pragma unroll
    for (int v = 0; v < V; ++v) dot[v] = 0.f;
    if (k < n) {
      const int t = k / Ns, c = k - t * Ns;
      const int cy = c / Mx, cx = c - cy * Mx;
      // bit (dx + 2) of vx: cx + dx inside the grid; likewise vy
      const uint32_t vx = (cx >= 2 ? 1u : 0u) | (cx >= 1 ? 2u : 0u) | 4u | (cx + 1 < Mx ? 8u : 0u) | (cx + 2 < Mx ? 16u : 0u);
      const uint32_t vy = (cy >= 2 ? 1u : 0u) | (cy >= 1 ? 2u : 0u) | 4u | (cy + 1 < Ny ? 8u : 0u) | (cy + 2 < Ny ? 16u : 0u);
      const uint32_t vt = (t > 0 ? 1u : 0u) | 2u | (t + 1 < T ? 4u : 0u);
      const float* cc = cf + c;
      const Cols<V>* xt = x + k;
      float acc[V];
      // a neighbour outside the grid counts with coefficient zero (on the node's own
      // value): no branches, so that the loads of a node overlap
      auto add = [&](int slot, int dx, int dy, int dt, bool in) {
        const float q = in ? cc[unsigned(slot) * unsigned(Ns)] : 0.f;
        const Cols<V> xv = xt[in ? dt * Ns + dy * Mx + dx : 0];
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] = fmaf(q, xv.v[v], acc[v]);
      };
      auto block25 = [&](int sb, int dt) {
        const bool vd = (vt >> (dt + 1)) & 1u;
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] = 0.f;
#pragma unroll
        for (int s = 0; s < 25; ++s) {
          const int dx = s % 5 - 2, dy = s / 5 - 2;
          add(sb + s, dx, dy, dt, vd && ((vx >> (dx + 2)) & (vy >> (dy + 2)) & 1u));
        }
      };
      auto block9 = [&](int s0, int dt) {
        const bool vd = (vt >> (dt + 1)) & 1u;
#pragma unroll
        for (int s = 0; s < 9; ++s) {
          const int dx = s % 3 - 1, dy = s / 3 - 1;
          add(s0 + s, dx, dy, dt, vd && ((vx >> (dx + 2)) & (vy >> (dy + 2)) & 1u));
        }
      };
      if (SEP) {
        // Q = Qt (x) Qs: Qt_tt (Qs x_t) + Qt_off (Qs x_(t-1) + Qs x_(t+1))
        float s[V];
        block25(25, 0);
#pragma unroll
        for (int v = 0; v < V; ++v) s[v] = (t == 0 || t == T - 1 ? qe : qm) * acc[v];
#pragma unroll
        for (int dt = -1; dt <= 1; dt += 2) {
          block25(25, dt);
#pragma unroll
          for (int v = 0; v < V; ++v) s[v] = fmaf(qo, acc[v], s[v]);
        }
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] = s[v];
      } else {
        block25(t == 0 && T > 1 ? 0 : 25, 0);
        add(68, 0, 0, 0, T > 1 && t < T - 1);
        if (T > 1) {
          block9(50, 1);
          block9(59, -1);
        }
      }
      const Cols<V> x0 = xt[0];
      if (o32) {
        const float q = o32[k];
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] = fmaf(q, x0.v[v], acc[v]);
      }
      Cols<V> r;
#pragma unroll
      for (int v = 0; v < V; ++v) {
        r.v[v] = acc[v];
        dot[v] = x0.v[v] * acc[v];
      }
      out[k] = r;
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const float w = warp_sum(dot[v]);
      if (lane == 0) part[int64_t(c0 + v) * gpad + g] = w;
    }
  }
}

// The same product for one column, a thread taking one cell through the time steps
// [t0, t1) of its CTA: the 43 coefficients (25 separable), which are the same at every
// interior step, stay in registers, and so do the 3 x 3 values around the cell that
// the next two steps read again, so that a step loads 25 values instead of 86.
// Every entry's products are added in spmv32_kernel's order.  With DOT (Ns % 32 = 0: a warp's
// nodes are a warp group) also the groups' sums of p . ap into part; otherwise
// group_dot_kernel forms them.
// Bound: latency, the loads in flight of 24 warps per SM (three CTAs; at two 175 us
// without spills, at four 152); the values two steps ahead are fetched to L2
// (130 us without).  At three CTAs its 80 registers spill 80 to 92 bytes (none separable).
// Measured at 400 x 400 x 48: 124 us, spmv32_kernel 177.
// Warps take runs of 32 cells as in Walk, with P runs per time step (the last one ragged).
struct CellWalk {
  int R, P, bx, steps;  // runs per grid row and per time step, CTAs per time step, time steps per CTA
};
constexpr int kAhead = 2;               // time steps between a value's fetch to L2 and its use
constexpr int kStepsCtas = 2 * 3 * 152;  // CTAs that the chunks of time steps are to leave
// Fewer steps per CTA than this do not pay for the coefficients' loads and, where the
// groups' sums take a launch of their own, for that launch (6 us at 10^6 nodes).
// Measured, against spmv32_kernel: 24 steps (400 x 400 x 48) 124 / 177 us, 5 (201 x 150 x
// 36, sums apart) 30.3 / 31.1, 4 (301 x 299 x 12, sums apart) 34 / 32, 1 (48 x 40 x 24) 6.3 / 6.1.
constexpr int kStepsMin = 5;
template <int SEP, int DOT>
__global__ void __launch_bounds__(256, 3) spmv32_steps_kernel(int Mx, int Ny, int T, float qe, float qm, float qo,
                                                              CellWalk wk, int lead, int gpad,
                                                              const float* __restrict__ cf,
                                                              const float* __restrict__ o32,
                                                              const float* __restrict__ pv, float* __restrict__ apv,
                                                              float* __restrict__ part) {
  const int Ns = Mx * Ny, n = Ns * T, lane = threadIdx.x & 31;
  const int by = int(blockIdx.x) / wk.bx, cta = int(blockIdx.x) - by * wk.bx;
  const int ry = cta / wk.R;
  const int a = (cta - ry * wk.R) + wk.R * (8 * ry + int(threadIdx.x >> 5));
  if (a >= wk.P) return;
  const int t0 = by * wk.steps, t1 = min(T, t0 + wk.steps);
  const int col = lead + int(blockIdx.y);
  const float* x = pv + int64_t(col) * n;
  float* out = apv + int64_t(col) * n;
  const bool mine = 32 * a + lane < Ns;  // the last run's other lanes repeat the last cell and store nothing
  const int c = min(32 * a + lane, Ns - 1);
  const int cy = c / Mx, cx = c - cy * Mx;
  // A neighbour outside the grid counts with coefficient zero on a value inside it.
  int xo[5], yo[5];
  bool xi[5], yi[5];
#pragma unroll
  for (int d = 0; d < 5; ++d) {
    xi[d] = cx + d - 2 >= 0 && cx + d - 2 < Mx;
    yi[d] = cy + d - 2 >= 0 && cy + d - 2 < Ny;
    xo[d] = xi[d] ? d - 2 : 0;
    yo[d] = yi[d] ? (d - 2) * Mx : 0;
  }
  const float* cc = cf + c;
  float qd[25], qn[9], qp[9], qs = 0.f;
  auto load_diag = [&](int sb) {
#pragma unroll
    for (int s = 0; s < 25; ++s) {
      const float q = cc[(sb + s) * Ns];
      qd[s] = (xi[s % 5] && yi[s / 5]) ? q : 0.f;
    }
  };
  if (SEP) {
    load_diag(25);
  } else {
    qs = cc[68 * Ns];
#pragma unroll
    for (int s = 0; s < 9; ++s) {
      const bool in = xi[s % 3 + 1] && yi[s / 3 + 1];
      const float u = cc[(50 + s) * Ns], w = cc[(59 + s) * Ns];
      qn[s] = in ? u : 0.f;
      qp[s] = in ? w : 0.f;
    }
  }
  auto ahead = [&](int t) {
    if (t >= T) return;
    asm volatile("prefetch.global.L2 [%0];" ::"l"(x + (t * Ns + c)));
    if (o32) asm volatile("prefetch.global.L2 [%0];" ::"l"(o32 + (t * Ns + c)));
  };
  // the 3 x 3 values around the cell at time t
  auto inner = [&](int t, float (&v)[9]) {
    const float* xt = x + (t * Ns + c);
#pragma unroll
    for (int s = 0; s < 9; ++s) v[s] = xt[yo[s / 3 + 1] + xo[s % 3 + 1]];
  };
  // the diagonal block (25 neighbours) at time t, whose inner values are u
  auto block25 = [&](int t, const float (&u)[9]) {
    const float* xt = x + (t * Ns + c);
    float acc = 0.f;
#pragma unroll
    for (int s = 0; s < 25; ++s) {
      const int dx = s % 5, dy = s / 5;
      const bool in3 = dx >= 1 && dx <= 3 && dy >= 1 && dy <= 3;
      acc = fmaf(qd[s], in3 ? u[in3 ? 3 * (dy - 1) + dx - 1 : 0] : xt[yo[dy] + xo[dx]], acc);
    }
    return acc;
  };
  auto finish = [&](int t, float x0, float acc) {
    const int k = t * Ns + c;
    if (o32) acc = fmaf(o32[k], x0, acc);
    if (mine) out[k] = acc;
    if (DOT) {
      const float w = warp_sum(__fmul_rn(x0, acc));
      if (lane == 0) part[int64_t(col) * gpad + t * wk.P + a] = w;
    }
  };
  if (SEP) {
    // Q = Qt (x) Qs: Qt_tt (Qs x_t) + Qt_off (Qs x_(t-1) + Qs x_(t+1)), every Qs x_t formed once
    float u[9], sp = 0.f;
    if (t0 > 0) {
      inner(t0 - 1, u);
      sp = block25(t0 - 1, u);
    }
    inner(t0, u);
    float x0 = u[4], sc = block25(t0, u);
    for (int t = t0; t < t1; ++t) {
      ahead(t + 1 + kAhead);
      float xn = 0.f, sn = 0.f;
      if (t + 1 < T) {
        inner(t + 1, u);
        xn = u[4];
        sn = block25(t + 1, u);
      }
      float acc = (t == 0 || t == T - 1 ? qe : qm) * sc;
      acc = fmaf(qo, sp, acc);
      acc = fmaf(qo, sn, acc);
      finish(t, x0, acc);
      sp = sc;
      sc = sn;
      x0 = xn;
    }
  } else {
    float pr[9], cu[9], nx[9];
    inner(t0, cu);
    if (t0 > 0) inner(t0 - 1, pr);
    for (int t = t0; t < t1; ++t) {
      if (t == t0 || t == 1) load_diag(t == 0 && T > 1 ? 0 : 25);
      ahead(t + kAhead);
      if (t + 1 < T) inner(t + 1, nx);
      float acc = block25(t, cu);
      if (t + 1 < T) {
        acc = fmaf(qs, cu[4], acc);
#pragma unroll
        for (int s = 0; s < 9; ++s) acc = fmaf(qn[s], nx[s], acc);
      }
      if (t > 0) {
#pragma unroll
        for (int s = 0; s < 9; ++s) acc = fmaf(qp[s], pr[s], acc);
      }
      finish(t, cu[4], acc);
#pragma unroll
      for (int s = 0; s < 9; ++s) {
        pr[s] = cu[s];
        cu[s] = nx[s];
      }
    }
  }
}

// The warp groups' sums of p . ap for the columns lead + y, one warp per group.  Bound:
// memory (8 bytes per node).
__global__ void __launch_bounds__(256) group_dot_kernel(int n, int ngroups, int lead, int gpad,
                                                        const float* __restrict__ pv, const float* __restrict__ apv,
                                                        float* __restrict__ part) {
  const int g = int(blockIdx.x) * 8 + int(threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (g >= ngroups) return;
  const int64_t col = lead + int(blockIdx.y);
  const int k = 32 * g + lane;
  const float w = warp_sum(k < n ? __fmul_rn(pv[col * n + k], apv[col * n + k]) : 0.f);
  if (lane == 0) part[col * gpad + g] = w;
}

// Diagonal of A at node (cell c, time t) from the FP32 coefficients.  The separable
// product rounds by itself, whatever is added to it, so that a column's bits do not depend
// on how many columns go together.
__device__ __forceinline__ float diag32(const float* __restrict__ cf, int Ns, int T, int sep, float qe, float qm,
                                        int c, int t) {
  if (sep) return __fmul_rn(t == 0 || t == T - 1 ? qe : qm, cf[int64_t(25 + 12) * Ns + c]);
  if (T == 1) return cf[int64_t(25 + 12) * Ns + c];
  if (t == 0) return cf[int64_t(12) * Ns + c] + cf[int64_t(68) * Ns + c];
  return cf[int64_t(25 + 12) * Ns + c] + (t < T - 1 ? cf[int64_t(68) * Ns + c] : 0.f);
}

// Elementwise step of column blockIdx.y (grid-stride over the nodes):
//   xc += alpha p, r -= alpha Ap   (alpha 0: no update)
//   mode 0: z = r;  mode 1: z = r / A_pp;  mode 2: z left to the G^T G kernel
// and the block's partial sums of r . z (mode < 2) into partA[col G + b] and of
// r . r into partB[col G + b].
// The sums are those of kElemBlocks blocks per column; the launch leaves out the blocks
// past the last node (G = gridDim.x of them run).
// Bound: memory (32 bytes per node and column with Jacobi and observations: x, r, p, Ap
// and the observation term read, x, r and z written, less z without a preconditioner) and, for one
// column, registers: at eight CTAs per SM its 32 spill 600 bytes of stores and 720 of loads a
// thread (60 us at 400 x 400 x 48, whose bytes need 36).
constexpr int kElemBlocks = 1216;  // 8 per SM
template <int V>
__global__ void __launch_bounds__(256, V == 1 ? 8 : 4) update32_kernel(int Ns, int T, int sep, float qe, float qm, int mode, int lead,
                                                       const float* __restrict__ cf, const float* __restrict__ o32,
                                                       float* __restrict__ xcv, float* __restrict__ rv,
                                                       const float* __restrict__ pv, const float* __restrict__ apv,
                                                       float* __restrict__ zv, const float* __restrict__ alpha,
                                                       double* __restrict__ partA, double* __restrict__ partB) {
  __shared__ float red[8];
  const int64_t n = int64_t(Ns) * T;
  const int c0 = lead + V * int(blockIdx.y);
  float a[V], srz[V], srr[V];
  bool step = false;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    a[v] = alpha[c0 + v];
    step |= a[v] != 0.f;
    srz[v] = srr[v] = 0.f;
  }
  Cols<V>* r = reinterpret_cast<Cols<V>*>(rv + c0 * n);
  Cols<V>* xc = reinterpret_cast<Cols<V>*>(xcv + c0 * n);
  Cols<V>* z = reinterpret_cast<Cols<V>*>(zv + c0 * n);
  const Cols<V>* p = reinterpret_cast<const Cols<V>*>(pv + c0 * n);
  const Cols<V>* ap = reinterpret_cast<const Cols<V>*>(apv + c0 * n);
  for (int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; k < n; k += int64_t(kElemBlocks) * blockDim.x) {
    Cols<V> rk = r[k];
    if (step) {
      Cols<V> xk = xc[k];
      const Cols<V> pk = p[k], ak = ap[k];
#pragma unroll
      for (int v = 0; v < V; ++v)
        if (a[v] != 0.f) {
          xk.v[v] = fmaf(a[v], pk.v[v], xk.v[v]);
          rk.v[v] = fmaf(-a[v], ak.v[v], rk.v[v]);
        }
      xc[k] = xk;
      r[k] = rk;
    }
#pragma unroll
    for (int v = 0; v < V; ++v) srr[v] = fmaf(rk.v[v], rk.v[v], srr[v]);
    if (mode < 2) {
      Cols<V> zk = rk;
      if (mode == 1) {
        const int t = int(k) / Ns, c = int(k) - t * Ns;  // node indices fit in 32 bits
        const float d = diag32(cf, Ns, T, sep, qe, qm, c, t) + (o32 ? o32[k] : 0.f);
#pragma unroll
        for (int v = 0; v < V; ++v) zk.v[v] = __fdividef(rk.v[v], d);
      }
      z[k] = zk;
#pragma unroll
      for (int v = 0; v < V; ++v) srz[v] = fmaf(rk.v[v], zk.v[v], srz[v]);
    }
  }
#pragma unroll
  for (int v = 0; v < V; ++v) {
    if (mode < 2) {
      const double b1 = block_sum(srz[v], red);
      if (threadIdx.x == 0) partA[int64_t(c0 + v) * gridDim.x + blockIdx.x] = b1;
    }
    const double b2 = block_sum(srr[v], red);
    if (threadIdx.x == 0) partB[int64_t(c0 + v) * gridDim.x + blockIdx.x] = b2;
  }
}

// Weights of G: compact (rows per cell and time class, observed rows through
// the bitmask and per-word ranks) or per node
struct GWeights {
  const float* w;
  const uint32_t* mask;  // compact, with observations: observed nodes have their own rows
  const int* rank;
  int nob, Ns, T, compact;
  // with mask: the nodes p whose row of G^T gathers from an observed node (bit p of
  // near, number of bits before each word in nrank) have that row written out,
  // near_w[o ncap + index]; without memory for it (near null) every weight is looked up
  const uint32_t* near;
  const int* nrank;
  const float* near_w;
  int ncap;
};

// Bits of the nodes whose G^T row gathers from an observed node: p = q + d for
// every observed q and offset d inside the grid.
__global__ void near_obs_kernel(const int* __restrict__ nodes, int nob, int Mx, int Ny, int T,
                                uint32_t* __restrict__ near) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nob) return;
  const int Ns = Mx * Ny, q = nodes[j];
  const int t = q / Ns, c = q - t * Ns, y = c / Mx, x = c - y * Mx;
  for (int o = 0; o < kOff; ++o) {
    const int dx = o % 3 - 1, dy = (o / 3) % 3 - 1, dt = o / 9 - 1;
    const int xp = x + dx, yp = y + dy, tp = t + dt;
    if (xp < 0 || xp >= Mx || yp < 0 || yp >= Ny || tp < 0 || tp >= T) continue;
    const int p = (tp * Ny + yp) * Mx + xp;
    atomicOr(&near[p >> 5], 1u << (p & 31));
  }
}

// rank[w] = number of set bits before word w (one block of 1024 threads)
__global__ void __launch_bounds__(1024) bit_rank_kernel(const uint32_t* __restrict__ bits, int nwords,
                                                        int* __restrict__ rank) {
  __shared__ int sums[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int base = 0;
  for (int w0 = 0; w0 < nwords; w0 += 1024) {
    const int i = w0 + tid, c = i < nwords ? __popc(bits[i]) : 0;
    int v = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, d);
      if (lane >= d) v += u;
    }
    if (lane == 31) sums[warp] = v;
    __syncthreads();
    int before = 0, all = 0;
    for (int q = 0; q < 32; ++q) {
      if (q < warp) before += sums[q];
      all += sums[q];
    }
    if (i < nwords) rank[i] = base + before + v - c;
    base += all;
    __syncthreads();
  }
}

__device__ __forceinline__ int time_class(int t, int T) { return t == 0 ? 0 : (t == T - 1 ? 2 : 1); }

// G(q, q + d_o) from the compact weights, q the node of cell cq at time tq
__device__ __forceinline__ float compact_weight(const GWeights& gw, int o, int cq, int tq, int q) {
  const uint32_t m = gw.mask[q >> 5], b = 1u << (q & 31);
  if (m & b) return gw.w[int64_t(3 * kOff) * gw.Ns + o * gw.nob + gw.rank[q >> 5] + __popc(m & (b - 1u))];
  return gw.w[int64_t(time_class(tq, gw.T) * kOff + o) * gw.Ns + cq];
}

// The rows of G^T next to observed nodes: near_w[o ncap + i] = weight with which
// node p gathers from q = p - d_o, 0 outside the grid
__global__ void near_rows_kernel(int Mx, int Ny, int T, GWeights gw, float* __restrict__ near_w) {
  const int Ns = Mx * Ny, n = Ns * T;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const uint32_t word = gw.near[p >> 5], bit = 1u << (p & 31);
  if (!(word & bit)) return;
  const int i = gw.nrank[p >> 5] + __popc(word & (bit - 1u));
  const int t = p / Ns, c = p - t * Ns, y = c / Mx, x = c - y * Mx;
  for (int o = 0; o < kOff; ++o) {
    const int dx = o % 3 - 1, dy = (o / 3) % 3 - 1, dt = o / 9 - 1;
    const int xq = x - dx, yq = y - dy, tq = t - dt;
    float v = 0.f;
    if (xq >= 0 && xq < Mx && yq >= 0 && yq < Ny && tq >= 0 && tq < T) {
      const int cq = yq * Mx + xq;
      v = compact_weight(gw, o, cq, tq, tq * Ns + cq);
    }
    near_w[int64_t(o) * gw.ncap + i] = v;
  }
}

// u = G r (TRANS 0) or z = G^T u with the warp groups' sums of r . z (TRANS 1) for
// the columns [lead + V y, + V), one thread per node and V columns; the rows of G
// come from the compact (COMPACT 1; 2: G^T without near_w) or per-node weights through L1 / L2.  Every
// row is one base, stride and neighbour shift per time offset, so that observed
// nodes, their neighbours and the boundary differ from the interior by a
// predicate per offset and not by another path (a warp holds several kinds).
// Offsets of the classes' rows fit in 32 bits (27 n < 2^31, checked by the caller; 54 Ns needs two
// time steps), the observed rows' start, 81 Ns, does not.  Bound: L1 / L2 loads.
// Measured at 200 x 200 x 24 with 1 % observed, 16 columns: G 101 us (413 with one
// column per thread), G^T 150 us (1,026: near an observed node, which is in nearly
// every warp, each of 27 weights was looked up through bitmask and rank).
template <int V, int TRANS, int COMPACT>
__global__ void __launch_bounds__(256, V == 1 ? 4 : 3) g32_kernel(int Mx, int Ny, int T, Walk wk, int lead, int gpad, GWeights gw,
                                                     const float* __restrict__ xv, float* __restrict__ outv,
                                                     const float* __restrict__ rv, float* __restrict__ part) {
  const int Ns = Mx * Ny, n = Ns * T, lane = threadIdx.x & 31;
  const int c0 = lead + V * int(blockIdx.y);
  const Cols<V>* x = reinterpret_cast<const Cols<V>*>(xv + int64_t(c0) * n);
  const Cols<V>* r = reinterpret_cast<const Cols<V>*>(rv + (TRANS ? int64_t(c0) * n : 0));
  Cols<V>* out = reinterpret_cast<Cols<V>*>(outv + int64_t(c0) * n);
  for (int j = 0; j < wk.steps; ++j) {
    const int g = walk_group(wk, j);
    if (g < 0) continue;
    const int p = 32 * g + lane;
    float dot[V];
#pragma unroll
    for (int v = 0; v < V; ++v) dot[v] = 0.f;
    if (p < n) {
      const int t = p / Ns, c = p - t * Ns;
      const int y = c / Mx, xx = c - y * Mx;
      // bit (d + 1) set: the neighbour at +d (G) or -d (G^T) is inside
      const int sg = TRANS ? -1 : 1;
      auto bits = [](int v, int lim, int sgn) {
        return (v - sgn >= 0 && v - sgn < lim ? 1u : 0u) | 2u | (v + sgn >= 0 && v + sgn < lim ? 4u : 0u);
      };
      const uint32_t bx = bits(xx, Mx, sg), by = bits(y, Ny, sg), bt = bits(t, T, sg);
      // weight of offset o: row[dt + 1][o stride - dy shift_y - dx shift_x]
      const float* row[3];
      int stride = 0, shift_y = 0, shift_x = 0;
      if (COMPACT == 0) {
        stride = n;
        shift_y = TRANS ? Mx : 0;
        shift_x = TRANS ? 1 : 0;
#pragma unroll
        for (int d = 0; d < 3; ++d) row[d] = gw.w + p - (TRANS ? (d - 1) * Ns : 0);
      } else if (COMPACT == 1) {
        const uint32_t* own = TRANS ? gw.near : gw.mask;  // nodes with a row of their own
        const uint32_t word = own ? own[p >> 5] : 0u, bit = 1u << (p & 31);
        if (word & bit) {
          const int i = (TRANS ? gw.nrank : gw.rank)[p >> 5] + __popc(word & (bit - 1u));
          stride = TRANS ? gw.ncap : gw.nob;
          row[0] = row[1] = row[2] = (TRANS ? gw.near_w : gw.w + int64_t(3 * kOff) * Ns) + i;
        } else {
          stride = Ns;
          shift_y = TRANS ? Mx : 0;
          shift_x = TRANS ? 1 : 0;
#pragma unroll
          for (int d = 0; d < 3; ++d) row[d] = gw.w + time_class(TRANS ? t - (d - 1) : t, T) * kOff * Ns + c;
        }
      }
      float acc[V];
#pragma unroll
      for (int v = 0; v < V; ++v) acc[v] = 0.f;
#pragma unroll
      for (int o = 0; o < kOff; ++o) {
        const int dx = o % 3 - 1, dy = (o / 3) % 3 - 1, dt = o / 9 - 1;
        // a neighbour outside the grid counts with weight zero (on the node's own value)
        const bool in = (bx >> (dx + 1)) & (by >> (dy + 1)) & (bt >> (dt + 1)) & 1u;
        const int d = in ? dt * Ns + dy * Mx + dx : 0;
        float wv = 0.f;
        if (COMPACT == 2) {
          if (in) wv = compact_weight(gw, o, c - dy * Mx - dx, t - dt, p - d);
        } else if (in) {
          wv = row[dt + 1][o * stride - dy * shift_y - dx * shift_x];
        }
        const Cols<V> xq = x[TRANS ? p - d : p + d];
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] = fmaf(wv, xq.v[v], acc[v]);
      }
      Cols<V> res;
#pragma unroll
      for (int v = 0; v < V; ++v) res.v[v] = acc[v];
      out[p] = res;
      if (TRANS) {
        const Cols<V> rp = r[p];
#pragma unroll
        for (int v = 0; v < V; ++v) dot[v] = rp.v[v] * acc[v];
      }
    }
    if (TRANS) {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const float w = warp_sum(dot[v]);
        if (lane == 0) part[int64_t(c0 + v) * gpad + g] = w;
      }
    }
  }
}

// ------------------------------------------------------------ IC(0)
// Incomplete Cholesky with the pattern of A's lower triangle in the natural
// node order (the baseline preconditioner of the PCG comparison).  The 21 lower
// neighbours of a node, ordered by increasing node index: dt = -1 (3 x 3),
// then dt = 0 with dy = -2, dy = -1 (dx -2..2 each) and dy = 0 (dx -2, -1).
// Every lower neighbour of node (x, y, t) lies on an earlier level of
// x + 3 y + 5 t, so the factorisation and the forward solve run level by
// level (one launch per level, the backward solve in reverse).  L is FP32, 22
// values per node: the 21 lower entries, then the diagonal.
constexpr int kIcLow = 21, kIcRow = 22;
struct IcTables {
  int dx[kIcLow], dy[kIcLow], dt[kIcLow];
  // for lower entry a: the common lower neighbours k of node i and of j = i + o_a
  // with k < j, as (index b of k in i's row, index c of k in j's row)
  int cstart[kIcLow + 1];
  int cb[512], cc[512];
};
__constant__ IcTables c_ic;

void ic_tables(IcTables* tb) {
  int m = 0;
  for (int dy = -1; dy <= 1; ++dy)
    for (int dx = -1; dx <= 1; ++dx) { tb->dx[m] = dx; tb->dy[m] = dy; tb->dt[m] = -1; ++m; }
  for (int dy = -2; dy <= -1; ++dy)
    for (int dx = -2; dx <= 2; ++dx) { tb->dx[m] = dx; tb->dy[m] = dy; tb->dt[m] = 0; ++m; }
  for (int dx = -2; dx <= -1; ++dx) { tb->dx[m] = dx; tb->dy[m] = 0; tb->dt[m] = 0; ++m; }
  auto find = [&](int dx, int dy, int dt) {
    for (int i = 0; i < kIcLow; ++i)
      if (tb->dx[i] == dx && tb->dy[i] == dy && tb->dt[i] == dt) return i;
    return -1;
  };
  int e = 0;
  for (int a = 0; a < kIcLow; ++a) {
    tb->cstart[a] = e;
    for (int b = 0; b < kIcLow; ++b) {
      // k = i + o_b must precede j = i + o_a and be a lower neighbour of j: o_b - o_a lower
      const int c = find(tb->dx[b] - tb->dx[a], tb->dy[b] - tb->dy[a], tb->dt[b] - tb->dt[a]);
      if (c >= 0) { tb->cb[e] = b; tb->cc[e] = c; ++e; }
    }
  }
  tb->cstart[kIcLow] = e;
}

// A(i, i + o) in FP32 from the coefficient copies (spatio-temporal layout)
__device__ __forceinline__ float aval32(const float* __restrict__ cf, const float* __restrict__ o32, int64_t Ns, int T,
                                        int k, int c, int t, int dx, int dy, int dt) {
  if (dt == -1) return cf[(59 + (dy + 1) * 3 + dx + 1) * Ns + c];
  if (dt == 1) return cf[(50 + (dy + 1) * 3 + dx + 1) * Ns + c];
  const int sb = (t == 0 && T > 1) ? 0 : 25;
  float v = cf[(sb + (dy + 2) * 5 + dx + 2) * Ns + c];
  if (dx == 0 && dy == 0) {
    if (T > 1 && t < T - 1) v += cf[68 * Ns + c];
    if (o32) v += o32[k];
  }
  return v;
}

// Node on level lev handled by thread e = (t, y): x = lev - 3 y - 5 t
__device__ __forceinline__ int ic_node(int lev, int e, int Mx, int Ny, int T, int* x, int* y, int* t) {
  if (e >= Ny * T) return -1;
  *t = e / Ny;
  *y = e - *t * Ny;
  *x = lev - 3 * *y - 5 * *t;
  if (*x < 0 || *x >= Mx) return -1;
  return (*t * Ny + *y) * Mx + *x;
}

// One level of the factorisation of A + shift diag(A); *bad counts pivots <= 0
__global__ void ic0_factor_kernel(int lev, int Mx, int Ny, int T, const float* __restrict__ cf,
                                  const float* __restrict__ o32, float shift, float* __restrict__ L,
                                  int* __restrict__ bad) {
  int x, y, t;
  const int i = ic_node(lev, blockIdx.x * blockDim.x + threadIdx.x, Mx, Ny, T, &x, &y, &t);
  if (i < 0) return;
  const int Ns = Mx * Ny, c = i - t * Ns;
  float* Li = L + int64_t(i) * kIcRow;
  bool in[kIcLow];
  float dsum = 0.f;
  for (int a = 0; a < kIcLow; ++a) {
    const int dx = c_ic.dx[a], dy = c_ic.dy[a], dt = c_ic.dt[a];
    in[a] = x + dx >= 0 && x + dx < Mx && y + dy >= 0 && y + dy < Ny && t + dt >= 0;
    if (!in[a]) { Li[a] = 0.f; continue; }
    const int j = i + dt * Ns + dy * Mx + dx;
    const float* Lj = L + int64_t(j) * kIcRow;
    float v = aval32(cf, o32, Ns, T, i, c, t, dx, dy, dt);
    for (int e = c_ic.cstart[a]; e < c_ic.cstart[a + 1]; ++e) {
      const int b = c_ic.cb[e];
      if (in[b]) v = fmaf(-Li[b], Lj[c_ic.cc[e]], v);  // b < a: Li[b] is final
    }
    const float lij = v / Lj[kIcLow];
    Li[a] = lij;
    dsum = fmaf(lij, lij, dsum);
  }
  float d = aval32(cf, o32, Ns, T, i, c, t, 0, 0, 0);
  d = d * (1.f + shift) - dsum;
  if (!(d > 0.f)) {
    atomicAdd(bad, 1);
    d = 1.f;
  }
  Li[kIcLow] = sqrtf(d);
}

// One level of L y = r (FWD) or L^T z = y (backward), column blockIdx.y
template <int FWD>
__global__ void ic0_solve_kernel(int lev, int Mx, int Ny, int T, const float* __restrict__ L,
                                 const float* __restrict__ in, float* __restrict__ out) {
  int x, y, t;
  const int i = ic_node(lev, blockIdx.x * blockDim.x + threadIdx.x, Mx, Ny, T, &x, &y, &t);
  if (i < 0) return;
  const int Ns = Mx * Ny, n = Ns * T;
  const int64_t off = int64_t(blockIdx.y) * n;
  float v = in[off + i];
#pragma unroll
  for (int a = 0; a < kIcLow; ++a) {
    const int dx = c_ic.dx[a], dy = c_ic.dy[a], dt = c_ic.dt[a];
    if (FWD) {
      if (x + dx < 0 || x + dx >= Mx || y + dy < 0 || y + dy >= Ny || t + dt < 0) continue;
      const int j = i + dt * Ns + dy * Mx + dx;
      v = fmaf(-L[int64_t(i) * kIcRow + a], out[off + j], v);
    } else {
      // upper neighbour j = i - o_a, whose row holds L(j, i) at index a
      if (x - dx < 0 || x - dx >= Mx || y - dy < 0 || y - dy >= Ny || t - dt >= T) continue;
      const int j = i - (dt * Ns + dy * Mx + dx);
      v = fmaf(-L[int64_t(j) * kIcRow + a], out[off + j], v);
    }
  }
  out[off + i] = v / L[int64_t(i) * kIcRow + kIcLow];
}

// partial sums of a . b per block and column (column blockIdx.y)
__global__ void __launch_bounds__(256) dot32c_kernel(const float* __restrict__ a, const float* __restrict__ b,
                                                     int n, double* __restrict__ part) {
  __shared__ float red[8];
  const int64_t off = int64_t(blockIdx.y) * n;
  float s = 0.f;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
    s = fmaf(a[off + k], b[off + k], s);
  const double bs = block_sum(s, red);
  if (threadIdx.x == 0) part[int64_t(blockIdx.y) * gridDim.x + blockIdx.x] = bs;
}

// Per-column scalars from partial sums in a fixed order: sum A over na block sums
// in partA, or (groupsA not null) over the blocks of eight warp groups each,
// ngroups groups in all at groupsA[col gpad ..]; sum B over nb block sums in partB.
// The blocks i, i + 256, ... are one chain of additions (256 chains, then a tree).
//   mode 0: pap = sum A;  alpha = rz / pap (0 if done or pap <= 0)
//   mode 1: rzn = sum A, rr = sum B;  beta = rzn / rz, rz = rzn
//   mode 2: rz = sum A, rr = sum B, beta = 0 (a new or replaced residual)
// gridDim.x (a power of two) CTAs share a column's chains, because an SM adds only
// two FP64 values per clock; the last of them to finish (`arrived`, left at zero)
// does the tree and the scalars.  Measured over 30,000 blocks: 12 us (94 with one CTA).
__global__ void __launch_bounds__(256) scal32_kernel(const float* __restrict__ groupsA, int ngroups, int gpad,
                                                     const double* __restrict__ partA, int na,
                                                     const double* __restrict__ partB, int nb, int mode,
                                                     const int* __restrict__ done, double* __restrict__ chains,
                                                     unsigned* __restrict__ arrived, double* __restrict__ rz,
                                                     double* __restrict__ rr, double* __restrict__ pap,
                                                     float* __restrict__ alpha, float* __restrict__ beta) {
  __shared__ double sh[2][256];
  __shared__ bool last;
  const int col = blockIdx.y, tid = threadIdx.x, Q = gridDim.x;
  const int W = 256 / Q, chain = tid & (W - 1), lane = tid / W;  // this CTA's chains Q-fold: blocks chain0 + chain + 256 j
  const int first = int(blockIdx.x) * W + chain;
  const int nblocks = groupsA ? (ngroups + 7) / 8 : na;
  const float4* ga = reinterpret_cast<const float4*>(groupsA + int64_t(col) * gpad);  // zero past the last group
  double s1 = 0.0, s2 = 0.0;
  // every CTA reads B's sums and the column's state (the last one's count), so that they do not
  // wait for the arrivals
  const bool over = mode != 2 && done[col];
  const double rz0 = mode != 2 ? rz[col] : 0.0;
  if (mode != 0)
    for (int i = tid; i < nb; i += 256) s2 += partB[int64_t(col) * nb + i];
  for (int j0 = 0; int(blockIdx.x) * W + 256 * j0 < nblocks; j0 += Q) {
    const int b = first + 256 * (j0 + lane);
    double s = 0.0;
    if (b < nblocks) {
      if (groupsA) {
        const float4 u = ga[2 * b], v = ga[2 * b + 1];
        s += u.x; s += u.y; s += u.z; s += u.w;
        s += v.x; s += v.y; s += v.z; s += v.w;
      } else {
        s = partA[int64_t(col) * na + b];
      }
    }
    sh[0][tid] = s;
    __syncthreads();
    if (tid < W)
      for (int q = 0; q < Q; ++q) s1 += sh[0][q * W + tid];
    __syncthreads();
  }
  if (Q > 1) {
    if (tid < W) {
      chains[int64_t(col) * 256 + first] = s1;
      __threadfence();
    }
    __syncthreads();
    if (tid == 0) last = atomicAdd(&arrived[col], 1u) == unsigned(Q - 1);
    __syncthreads();
    if (!last) return;
    __threadfence();
    s1 = __ldcg(chains + int64_t(col) * 256 + tid);
    if (tid == 0) arrived[col] = 0u;
  }
  sh[0][tid] = s1;
  sh[1][tid] = s2;
  __syncthreads();
  for (int k = 128; k > 0; k >>= 1) {
    if (tid < k) {
      sh[0][tid] += sh[0][tid + k];
      sh[1][tid] += sh[1][tid + k];
    }
    __syncthreads();
  }
  if (tid != 0) return;
  const double a = sh[0][0], b = sh[1][0];
  if (mode == 0) {
    pap[col] = a;
    alpha[col] = (!over && a > 0.0) ? float(rz0 / a) : 0.f;
  } else if (mode == 1) {
    beta[col] = (!over && rz0 != 0.0) ? float(a / rz0) : 0.f;
    rz[col] = a;
    rr[col] = b;
  } else {
    rz[col] = a;
    rr[col] = b;
    beta[col] = 0.f;
  }
}

//   p = z + beta p (finished columns unchanged), columns [lead + V y, + V)
template <int V>
__global__ void p32_kernel(float* __restrict__ pv, const float* __restrict__ zv, const float* __restrict__ beta,
                           const int* __restrict__ done, int64_t n, int lead) {
  const int c0 = lead + V * int(blockIdx.y);
  float b[V];
  bool run[V], any = false;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    b[v] = beta[c0 + v];
    run[v] = !done[c0 + v];
    any |= run[v];
  }
  if (!any) return;
  Cols<V>* p = reinterpret_cast<Cols<V>*>(pv + c0 * n);
  const Cols<V>* z = reinterpret_cast<const Cols<V>*>(zv + c0 * n);
  for (int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; k < n; k += int64_t(gridDim.x) * blockDim.x) {
    Cols<V> pk = p[k];
    const Cols<V> zk = z[k];
#pragma unroll
    for (int v = 0; v < V; ++v)
      if (run[v]) pk.v[v] = fmaf(b[v], pk.v[v], zk.v[v]);
    p[k] = pk;
  }
}

}  // namespace

int qsqrt_apply(Plan* p, int transpose, const double* x, double* y, int nrhs) {
  const int64_t len = int64_t(p->sym.n) * nrhs;
  if (len >= (int64_t(1) << 31)) return 1;
  const int Mx = p->sym.Mx, Ny = p->sym.Ny, T = p->sym.T;
  if (transpose)
    qsqrt_kernel<1><<<nblk(len), 256, 0, p->stream>>>(Mx, Ny, T, p->d_Ageo, p->d_A0geo, p->d_qs, p->model.V, p->cfac,
                                                      x, y, nrhs);
  else
    qsqrt_kernel<0><<<nblk(len), 256, 0, p->stream>>>(Mx, Ny, T, p->d_Ageo, p->d_A0geo, p->d_qs, p->model.V, p->cfac,
                                                      x, y, nrhs);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int pc_weights(Plan* p, int with_obs, double tau, const float* prm, float* w, float* act) {
  const int64_t n = p->sym.n;
  constexpr int kActSmem = (kNP + 128 * kAct) * int(sizeof(float));
  allow_smem<pc_forward_kernel>(kActSmem);
  pc_forward_kernel<<<nblk(n, 128), 128, act ? kActSmem : kNP * int(sizeof(float)), p->stream>>>(
      p->qstencil(), with_obs ? p->d_obs_cnt : nullptr, tau, prm, w, act);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int pc_grad(Plan* p, int with_obs, double tau, const float* prm, const float* w, const float* act, const double* z,
            int k, double* loss, float* grad) {
  const int64_t n = p->sym.n, len = n * k;
  if (len >= (int64_t(1) << 31)) return 1;  // the stencil kernels index entries in 32 bits
  const int nbw = int((n + kBwNodes - 1) / kBwNodes);
  // y, u, e, g1, g2 (n x k doubles each) + partial sums + per-node dout and block partials (as floats)
  const size_t dbl = size_t(5 * len) + size_t(kDotBlocks) * k + 8 + size_t(kColParts) * kNP + 32;
  const size_t flt = size_t(n) * kOff + size_t(nbw) * kNP;
  double* base = scratch(p, dbl + (flt + 1) / 2);
  if (!base) return 4;
  double *y = base, *u = y + len, *e = u + len, *g1 = e + len, *g2 = g1 + len, *part = g2 + len;
  double* sums = part + size_t(kDotBlocks) * k;
  double* colsums = sums + 8;
  unsigned* arrived = reinterpret_cast<unsigned*>(colsums + size_t(kColParts) * kNP);
  float* dout = reinterpret_cast<float*>(colsums + size_t(kColParts) * kNP + 32);
  float* bpart = dout + size_t(n) * kOff;
  const QStencil q = p->qstencil();
  const double* obs = with_obs ? p->d_obs_cnt : nullptr;
  cudaStream_t st = p->stream;
  pc_apply_kernel<1, double, double><<<nblk(len), 256, 0, st>>>(q, w, z, y, k);           // y = G^T z
  launch_spmv(q, obs, tau, y, u, k, st);                                   // u = A y
  pc_apply_kernel<0, double, double><<<nblk(len), 256, 0, st>>>(q, w, u, e, k);           // v = G u
  pc_sub_kernel<<<nblk(len), 256, 0, st>>>(z, e, len);                     // e = z - v
  pc_apply_kernel<1, double, double><<<nblk(len), 256, 0, st>>>(q, w, e, g1, k);          // G^T e
  launch_spmv(q, obs, tau, g1, g2, k, st);                                 // g = A G^T e
  // loss = ||e||^2 / (n k): one column of length n k
  pc_dot_partial_kernel<<<kDotBlocks, 256, 0, st>>>(e, e, len, 1, part);
  pc_dot_final_kernel<<<1, 64, 0, st>>>(part, kDotBlocks, 1, sums);
  const double scale = -2.0 / double(len);
  if (k == 4) pc_wgrad_kernel<4><<<nblk(n, 128), 128, 0, st>>>(q, z, e, u, g2, k, scale, act, dout);
  else pc_wgrad_kernel<0><<<nblk(n, 128), 128, 0, st>>>(q, z, e, u, g2, k, scale, act, dout);
  const size_t smem = sizeof(float) * (kHid * kHid + kOff * kHid + kBwNodes * (kFeat + 4 * kHid + kOff));
  allow_smem<pc_backward_kernel>(int(smem));
  pc_backward_kernel<<<nbw, kBwThreads, smem, st>>>(n, prm, act, dout, bpart);
  cudaMemsetAsync(arrived, 0, 32 * sizeof(double), st);
  pc_colsum_kernel<<<dim3(nblk(kNP, 128), kColParts), 128, 0, st>>>(bpart, nbw, colsums, arrived, grad);
  double h = 0.0;
  cudaMemcpyAsync(&h, sums, sizeof(double), cudaMemcpyDeviceToHost, st);
  if (cudaStreamSynchronize(st) != cudaSuccess) return 2;
  *loss = h / double(len);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int pc_adam(const float* g, float* prm, float* m, float* v, int n, float lr, float b1, float b2, float eps, int t,
            cudaStream_t st) {
  const float c1 = 1.f - powf(b1, float(t)), c2 = 1.f - powf(b2, float(t));
  adam_kernel<<<nblk(n), 256, 0, st>>>(prm, g, m, v, n, lr, b1, b2, eps, c1, c2);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int jacobi_smooth(Plan* p, int with_obs, double tau, double omega, int sweeps, double* z, int nrhs) {
  const int64_t n = p->sym.n, len = n * nrhs;
  double* base = scratch(p, size_t(len) + size_t(kDotBlocks) * nrhs + size_t(nrhs) + size_t(n));
  if (!base) return 4;
  double *az = base, *part = az + len, *ss = part + size_t(kDotBlocks) * nrhs, *wd = ss + nrhs;
  const QStencil q = p->qstencil();
  const double* obs = with_obs ? p->d_obs_cnt : nullptr;
  if (q.sep || sweeps == 1) {  // a single sweep: one launch fewer than with weights and a copy back
    for (int it = 0; it < sweeps; ++it) {
      launch_spmv(q, obs, tau, z, az, nrhs, p->stream);
      jacobi_sweep_kernel<<<nblk(len), 256, 0, p->stream>>>(q, obs, tau, omega, az, z, nrhs);
    }
  } else {
    // one launch per sweep, from z to the scratch block and back
    jacobi_weight_kernel<<<nblk(n), 256, 0, p->stream>>>(q, obs, tau, omega, wd);
    double *from = z, *to = az;
    for (int it = 0; it < sweeps; ++it) {
      launch_jacobi_sweep(q, obs, tau, wd, from, to, nrhs, p->stream);
      std::swap(from, to);
    }
    if (from != z) cudaMemcpyAsync(z, from, size_t(len) * sizeof(double), cudaMemcpyDeviceToDevice, p->stream);
  }
  col_dots(p, z, z, nrhs, part, ss);
  col_scale_kernel<<<nblk(len), 256, 0, p->stream>>>(z, ss, n, nrhs);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

float* scratch32(Plan* p, size_t elems) {
  if (elems > p->pc32_cap) {
    cudaFree(p->d_pc32);
    p->d_pc32 = nullptr;
    p->pc32_cap = 0;
    if (cudaMalloc(&p->d_pc32, elems * sizeof(float)) != cudaSuccess) return nullptr;
    p->pc32_cap = elems;
  }
  return static_cast<float*>(p->d_pc32);
}

// Compact weights start with a 4-int header (magic, observed rows included,
// observation-set version, number of observed rows) so that a solve can check
// that they belong to its observation set; the rows follow.
constexpr int kCompactHeader = 4;
constexpr int kCompactMagic = 0x53504345;

int64_t pc_compact_floats(const Plan* p) {
  return kCompactHeader + int64_t(kOff) * (3 * int64_t(p->sym.Mx) * p->sym.Ny + p->nob);
}

int pc_weights_compact(Plan* p, int with_obs, double tau, const float* prm, float* w) {
  const int Ns = p->sym.Mx * p->sym.Ny;
  const int nob = with_obs ? p->nob : 0;
  const int64_t rows = 3 * int64_t(Ns) + nob;
  static thread_local int head[kCompactHeader];
  head[0] = kCompactMagic;
  head[1] = with_obs ? 1 : 0;
  head[2] = p->obs_version;
  head[3] = nob;
  cudaMemcpyAsync(w, head, sizeof(head), cudaMemcpyHostToDevice, p->stream);
  pc_forward_compact_kernel<<<nblk(rows, 128), 128, 0, p->stream>>>(p->qstencil(), with_obs ? p->d_obs_cnt : nullptr,
                                                                    tau, p->d_obs_nodes, nob, prm,
                                                                    w + kCompactHeader);
  // the header copy reads host memory asynchronously: finish before it can change
  return cudaStreamSynchronize(p->stream) == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : 2;
}

// Reliable-update PCG: the recursive FP32 residual is replaced by the true
// FP64 one (and the FP32 correction added into the FP64 solution) whenever it
// has fallen by this factor since the last replacement, reaches the tolerance,
// or kReplaceEvery iterations have passed.
constexpr double kReplaceDrop = 0.1;
constexpr int kReplaceEvery = 64;

// Whether a solve's columns go in groups of 4, 2 and 1 or each by itself (a column's bits are the
// same).  Every width is a launch of its own in each step, and widths follow one another: with two
// or three of them a small solve is faster by single columns, in one launch.  Measured (Jacobi,
// groups / single columns, us a solve): 3 columns at 40 x 30 x 8 3,754 / 2,448, at 200 x 200 x 24
// 11,155 / 10,381; 6 at 90 x 70 x 12 4,663 / 3,913, at 160 x 150 x 16 7,943 / 8,332; 7 at 110 x 100 x 16
// 8,285 / 6,644; 17 at 90 x 70 x 12 5,940 / 6,163.
bool columns_grouped(int64_t n, int nrhs) {
  const int widths = (nrhs >= 4) + ((nrhs & 2) != 0) + (nrhs & 1);
  if (widths == 1) return true;
  if (nrhs == 3) return false;
  return n * nrhs > int64_t(1) << (widths == 2 ? 19 : 21);
}

int pcg_solve(Plan* p, int with_obs, double tau, int kind, const float* w, const double* b, double* x, int nrhs,
              double tol, int maxit, int check_every, int* iters, double* relres) {
  const int64_t n = p->sym.n, len = n * nrhs;
  // the stencil kernels index nodes and the weights of one class (27 n at most) in 32 bits
  if (len >= (int64_t(1) << 31) || int64_t(p->sym.n) * kOff >= (int64_t(1) << 31) || nrhs > 65535) return 1;
  const int Mx = p->sym.Mx, Ny = p->sym.Ny, Ns = Mx * Ny, T = p->sym.T;
  cudaStream_t st = p->stream;
  const int nsp = nblk(n, 256);  // blocks of 256 consecutive nodes (dot products)
  const int ngroups = nblk(n, 32), gpad = 8 * nsp;
  const int nel = std::min(int(kElemBlocks), nsp);  // elementwise blocks with nodes
  const int na_max = std::max(nsp, int(kElemBlocks));
  const int packed = kind != 4 && columns_grouped(n, nrhs) ? 1 : 0;
  // FP64: true residual (row-major), block partials, per-column scalars
  const size_t need64 = size_t(len) + size_t(nrhs) * (na_max + kElemBlocks) + size_t(kDotBlocks) * nrhs +
                        size_t(8 * nrhs) + size_t(nrhs) + size_t(257) * nrhs;
  double* base = scratch(p, need64);
  // FP32: r, z, p, Ap, x correction, G r (grouped columns); coefficients; observation
  // term; warp-group sums; alpha, beta; rows of G^T next to observed nodes
  const bool near_bits = kind == 3 && with_obs;  // G^T needs the nodes next to observed ones
  const size_t nwords = size_t((n + 31) / 32);
  const int64_t ncap = near_bits ? std::min<int64_t>(n, int64_t(kOff) * p->nob) : 0;
  auto pad4 = [](size_t e) { return (e + 3) & ~size_t(3); };  // 16-byte sections
  const size_t vlen = pad4(size_t(len));  // a group of columns then starts at a multiple of its width
  const size_t need32 = 6 * vlen + size_t(nrhs) * gpad + pad4(size_t(kCoef32) * Ns) + pad4(size_t(n)) +
                        pad4(size_t(2 * nrhs)) + (kind == 4 ? pad4(size_t(kIcRow) * n) : 0);
  // the rows of G^T next to observed nodes (27 floats for up to every node): a solve that has no
  // memory for them looks the weights up, with the same result
  bool near_table = near_bits;
  float* b32 = scratch32(p, need32 + (near_table ? 2 * pad4(nwords) + size_t(kOff) * ncap : 0));
  if (!b32 && near_table) {
    cudaGetLastError();
    near_table = false;
    b32 = scratch32(p, need32);
  }
  if (!base || !b32) return 4;
  double* r64 = base;
  double* partA = r64 + len;
  double* partB = partA + size_t(nrhs) * na_max;
  double* part64 = partB + size_t(nrhs) * kElemBlocks;
  double* sc = part64 + size_t(kDotBlocks) * nrhs;
  double *rz = sc, *pap = sc + nrhs, *rr = sc + 2 * nrhs, *bb = sc + 3 * nrhs, *rrt = sc + 4 * nrhs;
  int* done = reinterpret_cast<int*>(sc + 8 * nrhs);
  double* chains = sc + 9 * nrhs;  // 256 per column
  unsigned* arrived = reinterpret_cast<unsigned*>(chains + size_t(256) * nrhs);
  float *r32 = b32, *z32 = r32 + vlen, *p32 = z32 + vlen, *ap32 = p32 + vlen, *xc32 = ap32 + vlen, *u32 = xc32 + vlen;
  float* gsum = u32 + vlen;  // warp groups' sums of a dot product, per column
  float* cf = gsum + size_t(nrhs) * gpad;
  float* o32 = cf + pad4(size_t(kCoef32) * Ns);
  float* alpha = o32 + pad4(size_t(n));
  float* beta = alpha + nrhs;
  float* Lic = alpha + pad4(size_t(2 * nrhs));  // IC(0) factor (kind 4)
  uint32_t* near = reinterpret_cast<uint32_t*>(Lic + (kind == 4 ? pad4(size_t(kIcRow) * n) : 0));
  int* nrank = reinterpret_cast<int*>(near + (near_table ? pad4(nwords) : 0));
  float* near_w = reinterpret_cast<float*>(nrank + (near_table ? pad4(nwords) : 0));
  const QStencil q = p->qstencil();
  const double* obs = with_obs ? p->d_obs_cnt : nullptr;
  const int sep = q.sep;
  const float qe = float(q.qt_end), qm = float(q.qt_mid), qo = float(q.qt_off);
  const int mode = kind == 0 ? 0 : (kind == 1 ? 1 : 2);  // 2: z from a separate preconditioner pass
  // IC(0) of the spatio-temporal stencil; its lower-neighbour order needs Mx >= 5, Ny >= 4
  if (kind == 4 && (q.sep || T < 2 || Mx < 5 || Ny < 4)) return 8;
  if (kind == 3) {
    // compact weights hold observed rows for the observation set they were computed with
    int head[kCompactHeader] = {0, 0, 0, 0};
    if (cudaMemcpyAsync(head, w, sizeof(head), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      return 2;
    const bool ok = head[0] == kCompactMagic && head[1] == (with_obs ? 1 : 0) &&
                    (!with_obs || (head[2] == p->obs_version && head[3] == p->nob));
    if (!ok) return 7;
    w += kCompactHeader;
  }
  GWeights gw{w, near_bits ? p->d_obs_mask : nullptr, p->d_obs_rank, p->nob, Ns, T, kind == 3 ? 1 : 0,
              near_table ? near : nullptr, nrank, near_w, int(ncap)};
  if (near_table) {
    cudaMemsetAsync(near, 0, nwords * sizeof(uint32_t), st);
    if (p->nob > 0) near_obs_kernel<<<nblk(p->nob), 256, 0, st>>>(p->d_obs_nodes, p->nob, Mx, Ny, T, near);
    bit_rank_kernel<<<1, 1024, 0, st>>>(near, int(nwords), nrank);
    near_rows_kernel<<<nblk(n), 256, 0, st>>>(Mx, Ny, T, gw, near_w);
  }
  cudaMemsetAsync(gsum, 0, size_t(nrhs) * gpad * sizeof(float), st);
  cudaMemsetAsync(arrived, 0, size_t(nrhs) * sizeof(unsigned), st);
  coef32_kernel<<<nblk(Ns, 128), 128, 0, st>>>(q, cf);
  if (obs) obs32_kernel<<<nblk(n), 256, 0, st>>>(obs, tau, o32, n);
  const float* o = obs ? o32 : nullptr;
  // f(IntC<V>, first column, groups) for the columns in groups of V = 4, 2, 1
  auto by_groups = [&](auto&& f) {
    const int n4 = packed ? nrhs & ~3 : 0, n2 = packed ? nrhs & 2 : 0, n1 = nrhs - n4 - n2;
    if (n4) f(IntC<4>{}, 0, n4 / 4);
    if (n2) f(IntC<2>{}, n4, 1);
    if (n1) f(IntC<1>{}, n4 + n2, n1);
  };
  // time steps per CTA of the per-node kernels: as many as leave the GPU two waves
  // of CTAs (four per SM)
  auto walk = [&](int groups, dim3* grid) {
    Walk wk;
    wk.P = std::max(1, (Ns + 16) / 32);
    wk.R = std::max(1, std::min(wk.P, (Mx + 16) / 32));
    wk.ngroups = ngroups;
    wk.rows8 = ((wk.P + wk.R - 1) / wk.R + 7) / 8;
    wk.bx = wk.R * wk.rows8;
    const int nb = (ngroups + wk.P - 1) / wk.P;
    wk.steps = 8;
    while (wk.steps > 1 && int64_t(wk.bx) * ((nb + wk.steps - 1) / wk.steps) * groups < 2 * 4 * 152) wk.steps /= 2;
    *grid = dim3(wk.bx * ((nb + wk.steps - 1) / wk.steps), groups);
    return wk;
  };
  const int nlev = (Mx - 1) + 3 * (Ny - 1) + 5 * (T - 1) + 1;
  const dim3 glev(nblk(int64_t(Ny) * T, 128), nrhs);
  if (kind == 4) {
    // IC(0) of A + shift diag(A), the shift raised until no pivot breaks down
    static IcTables tables;
    static const bool tables_ready = (ic_tables(&tables), true);
    (void)tables_ready;
    if (cudaMemcpyToSymbolAsync(c_ic, &tables, sizeof(IcTables), 0, cudaMemcpyHostToDevice, st) != cudaSuccess)
      return 2;
    int* bad = reinterpret_cast<int*>(alpha);  // alpha is set before its first use
    const float shifts[] = {0.f, 1e-3f, 1e-2f, 1e-1f, 1.f};
    bool ok = false;
    for (float sh : shifts) {
      cudaMemsetAsync(bad, 0, sizeof(int), st);
      for (int lev = 0; lev < nlev; ++lev)
        ic0_factor_kernel<<<nblk(int64_t(Ny) * T, 128), 128, 0, st>>>(lev, Mx, Ny, T, cf, o, sh, Lic, bad);
      int hb = 0;
      if (cudaMemcpyAsync(&hb, bad, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
          cudaStreamSynchronize(st) != cudaSuccess)
        return 2;
      if (hb == 0) { ok = true; break; }
    }
    if (!ok) return 9;
  }
  // z = M r with the partial sums of r . z and r . r, after the update of r by alpha
  auto update_precond = [&]() {
    by_groups([&](auto vw, int lead, int groups) {
      constexpr int V = decltype(vw)::value;
      update32_kernel<V><<<dim3(nel, groups), 256, 0, st>>>(Ns, T, sep, qe, qm, mode, lead, cf, o, xc32, r32, p32, ap32,
                                                            z32, alpha, partA, partB);
      if (mode != 2 || kind == 4) return;
      dim3 grid;
      const Walk wk = walk(groups, &grid);
      if (kind == 3) {
        g32_kernel<V, 0, 1><<<grid, 256, 0, st>>>(Mx, Ny, T, wk, lead, gpad, gw, r32, u32, nullptr, nullptr);
        if (near_bits && !near_table)
          g32_kernel<V, 1, 2><<<grid, 256, 0, st>>>(Mx, Ny, T, wk, lead, gpad, gw, u32, z32, r32, gsum);
        else
          g32_kernel<V, 1, 1><<<grid, 256, 0, st>>>(Mx, Ny, T, wk, lead, gpad, gw, u32, z32, r32, gsum);
      } else {
        g32_kernel<V, 0, 0><<<grid, 256, 0, st>>>(Mx, Ny, T, wk, lead, gpad, gw, r32, u32, nullptr, nullptr);
        g32_kernel<V, 1, 0><<<grid, 256, 0, st>>>(Mx, Ny, T, wk, lead, gpad, gw, u32, z32, r32, gsum);
      }
    });
    if (kind == 4) {
      for (int lev = 0; lev < nlev; ++lev)
        ic0_solve_kernel<1><<<glev, 128, 0, st>>>(lev, Mx, Ny, T, Lic, r32, u32);
      for (int lev = nlev - 1; lev >= 0; --lev)
        ic0_solve_kernel<0><<<glev, 128, 0, st>>>(lev, Mx, Ny, T, Lic, u32, z32);
      dot32c_kernel<<<dim3(nsp, nrhs), 256, 0, st>>>(r32, z32, int(n), partA);
    }
  };
  // r . z: block sums of the update (none, Jacobi) or of IC(0)'s dot product, else G^T's group sums
  const int na = mode == 2 ? nsp : nel;
  const float* gz = mode == 2 && kind != 4 ? gsum : nullptr;
  // CTAs per column of the scalar kernel: one per block of each chain, up to 64.  Measured with Jacobi,
  // one column, at one CTA per 2 / 1 / 0.5 blocks: 130 x 120 x 16 3,881 / 3,604 / 3,606 us a solve,
  // 200 x 200 x 16 4,648 / 4,506 / 4,573, 400 x 400 x 48 25.4 / 25.4 / 25.4 ms.
  auto scalars = [&](const float* groups, int na_, int nb_, int what) {
    int Q = 1;
    while (Q < 64 && (groups ? nsp : na_) > 256 * Q) Q *= 2;
    scal32_kernel<<<dim3(Q, nrhs), 256, 0, st>>>(groups, ngroups, gpad, partA, na_, partB, nb_, what, done, chains,
                                                 arrived, rz, rr, pap, alpha, beta);
  };
  auto new_direction = [&]() {  // p = z + beta p
    by_groups([&](auto vw, int lead, int groups) {
      p32_kernel<decltype(vw)::value><<<dim3(nel, groups), 256, 0, st>>>(p32, z32, beta, done, n, lead);
    });
  };
  // a new residual r32: z = M r, rz = r . z (p unchanged)
  auto restart = [&]() {
    cudaMemsetAsync(alpha, 0, size_t(nrhs) * sizeof(float), st);
    update_precond();
    scalars(gz, na, nel, 2);
  };
  auto true_residual = [&]() {
    launch_spmv(q, obs, tau, x, r64, nrhs, st);
    pc_sub_kernel<<<nblk(len), 256, 0, st>>>(b, r64, len);
    col_dots(p, r64, r64, nrhs, part64, rrt);
  };
  cudaMemsetAsync(x, 0, size_t(len) * sizeof(double), st);
  cudaMemsetAsync(xc32, 0, size_t(len) * sizeof(float), st);
  cudaMemsetAsync(p32, 0, size_t(len) * sizeof(float), st);
  col_dots(p, b, b, nrhs, part64, bb);
  std::vector<double> hb(nrhs), hr(nrhs), href(nrhs);
  std::vector<int> hd(nrhs, 0);
  cudaMemcpyAsync(hb.data(), bb, nrhs * sizeof(double), cudaMemcpyDeviceToHost, st);
  if (cudaStreamSynchronize(st) != cudaSuccess) return 2;
  for (int c = 0; c < nrhs; ++c)
    if (!(hb[c] > 0.0)) hd[c] = 1;  // a zero right-hand side is solved by x = 0
  cudaMemcpyAsync(done, hd.data(), nrhs * sizeof(int), cudaMemcpyHostToDevice, st);
  href = hb;
  to32cm_kernel<<<nblk(len), 256, 0, st>>>(b, r32, n, nrhs, packed);
  restart();
  new_direction();  // p = z
  const double tol2 = tol * tol;
  const int every = std::max(1, std::min(check_every, 4));
  int it = 0, last_rep = 0;
  bool all_done = false, fresh = false;  // fresh: x holds every correction and rrt is its true residual
  for (int c = 0; c < nrhs; ++c) all_done = (c == 0 || all_done) && hd[c];
  while (it < maxit && !all_done) {
    by_groups([&](auto vw, int lead, int groups) {
      constexpr int V = decltype(vw)::value;
      dim3 grid;
      if (V == 1) {
        CellWalk cw;
        cw.P = (Ns + 31) / 32;
        cw.R = std::max(1, std::min(cw.P, (Mx + 16) / 32));
        cw.bx = cw.R * (((cw.P + cw.R - 1) / cw.R + 7) / 8);
        // few chunks of time steps, but kStepsCtas CTAs
        const int64_t per = int64_t(cw.bx) * groups;
        const int chunks = int(std::min<int64_t>(T, (kStepsCtas + per - 1) / per));
        cw.steps = (T + chunks - 1) / chunks;
        if (cw.steps >= kStepsMin) {
          grid = dim3(cw.bx * ((T + cw.steps - 1) / cw.steps), groups);
          auto product = [&](auto sp, auto dot) {
            spmv32_steps_kernel<decltype(sp)::value, decltype(dot)::value><<<grid, 256, 0, st>>>(
                Mx, Ny, T, qe, qm, qo, cw, lead, gpad, cf, o, p32, ap32, gsum);
          };
          const bool dot = Ns % 32 == 0;
          if (sep && dot) product(IntC<1>{}, IntC<1>{});
          else if (sep) product(IntC<1>{}, IntC<0>{});
          else if (dot) product(IntC<0>{}, IntC<1>{});
          else product(IntC<0>{}, IntC<0>{});
          if (!dot)
            group_dot_kernel<<<dim3((ngroups + 7) / 8, groups), 256, 0, st>>>(int(n), ngroups, lead, gpad, p32, ap32,
                                                                              gsum);
          return;
        }
      }
      const Walk wk = walk(groups, &grid);
      if (sep)
        spmv32_kernel<V, 1><<<grid, 256, 0, st>>>(Mx, Ny, T, qe, qm, qo, wk, lead, gpad, cf, o, p32, ap32, gsum);
      else
        spmv32_kernel<V, 0><<<grid, 256, 0, st>>>(Mx, Ny, T, qe, qm, qo, wk, lead, gpad, cf, o, p32, ap32, gsum);
    });
    scalars(gsum, 0, 0, 0);
    update_precond();
    scalars(gz, na, nel, 1);
    new_direction();
    ++it;
    fresh = false;
    if (it % every != 0 && it != maxit) continue;
    cudaMemcpyAsync(hr.data(), rr, nrhs * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return 2;
    bool replace = it == maxit || it - last_rep >= kReplaceEvery;
    for (int c = 0; c < nrhs && !replace; ++c)
      if (!hd[c] && (hr[c] <= kReplaceDrop * kReplaceDrop * href[c] || hr[c] <= tol2 * hb[c])) replace = true;
    if (!replace) continue;
    acc64cm_kernel<<<nblk(len), 256, 0, st>>>(x, xc32, n, nrhs, packed);
    true_residual();
    cudaMemcpyAsync(hr.data(), rrt, nrhs * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return 2;
    fresh = true;
    last_rep = it;
    all_done = true;
    for (int c = 0; c < nrhs; ++c) {
      if (!hd[c] && hr[c] <= tol2 * hb[c]) hd[c] = 1;
      all_done = all_done && hd[c];
      href[c] = hr[c];
    }
    if (all_done) break;
    cudaMemcpyAsync(done, hd.data(), nrhs * sizeof(int), cudaMemcpyHostToDevice, st);
    // continue from the true residual (p kept)
    to32cm_kernel<<<nblk(len), 256, 0, st>>>(r64, r32, n, nrhs, packed);
    restart();
  }
  if (!fresh) {
    acc64cm_kernel<<<nblk(len), 256, 0, st>>>(x, xc32, n, nrhs, packed);
    true_residual();
    cudaMemcpyAsync(hr.data(), rrt, nrhs * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return 2;
  }
  double worst = 0.0;
  for (int c = 0; c < nrhs; ++c) worst = std::max(worst, hb[c] > 0.0 ? sqrt(hr[c] / hb[c]) : 0.0);
  *iters = it;
  *relres = worst;
  return cudaGetLastError() == cudaSuccess ? (worst <= tol ? 0 : 6) : 2;
}

}  // namespace spde
