// Batched dense kernels of the multifrontal factorisation, selected inversion
// and solves.  Every launch walks a task list prepared once per lattice by the
// symbolic phase, so fronts of very different sizes share one launch.
//
// This file holds the SIMT kernels (FP64 "plain" path, and the FP32 path on
// tiles the tensor-core kernel does not take).
#include <cuda_runtime.h>
#include <math.h>
#include <stdlib.h>

#include "kernels.cuh"
#include "tc_common.cuh"

namespace spde {

// --------------------------------------------------------------------- GEMM
// Tiled product on the CUDA cores, FP64 storage.  A, B and C may alias (in-place
// triangular solves): every block reads all of its A and B tiles before its
// epilogue writes C, and blocks own disjoint C tiles.
template <int MODE, int AL, int BL>
__global__ void __launch_bounds__(256) gemm64_kernel(const GemmTask* __restrict__ tasks, const double* Ab,
                                                     const double* Bb, double* Cb) {
  using T = double;
  constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;
  __shared__ T As[BK][BM + 4];
  __shared__ T Bs[BK][BN + 4];
  const GemmTask tk = tasks[blockIdx.x];
  const T* A = Ab + tk.a;
  const T* B = Bb + tk.b;
  T* Cp = Cb + tk.c;
  const int tid = threadIdx.x;
  chain_wait();
  const int tx = tid % (BN / TN);  // column group
  const int ty = tid / (BN / TN);  // row group
  T acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = T(0);
  for (int k0 = 0; k0 < tk.k; k0 += BK) {
    // A tile: BM x BK
    for (int e = tid; e < BM * BK; e += 256) {
      int i, kk;
      if (AL == kRow) { kk = e % BK; i = e / BK; } else { i = e % BM; kk = e / BM; }
      T v = T(0);
      if (i < tk.m && k0 + kk < tk.k)
        v = (AL == kRow) ? A[int64_t(i) * tk.lda + k0 + kk] : A[int64_t(k0 + kk) * tk.lda + i];
      As[kk][i] = v;
    }
    for (int e = tid; e < BN * BK; e += 256) {
      int j, kk;
      if (BL == kRow) { kk = e % BK; j = e / BK; } else { j = e % BN; kk = e / BN; }
      T v = T(0);
      if (j < tk.n && k0 + kk < tk.k)
        v = (BL == kRow) ? B[int64_t(j) * tk.ldb + k0 + kk] : B[int64_t(k0 + kk) * tk.ldb + j];
      Bs[kk][j] = v;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      T a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = Bs[kk][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    int r = ty * TM + i;
    if (r >= tk.m) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      int c = tx * TN + j;
      if (c >= tk.n) continue;
      T* dst = Cp + int64_t(r) * tk.ldc + c;
      if (MODE == kSub) *dst -= acc[i][j];
      else if (MODE == kStore) *dst = acc[i][j];
      else if (MODE == kNegStore) *dst = -acc[i][j];
      else *dst += acc[i][j];
    }
  }
}

// The same in FP32: 128 x 128 tiles, 8 x 8 entries per thread, K in chunks of 32
// copied asynchronously into one of two shared-memory buffers while the other is
// used.  An operand lies in shared memory as in memory: rows of 32 k values (row
// layout, read two k values at a time) or, per k, rows side by side (column layout);
// a warp computes 32 x 64 entries, warps outside the task's rows or columns skip the
// arithmetic.  Every entry adds its products in the order of k.  Same aliasing rule
// as above.  Bound: the FP32 pipe for many tiles, latency for few.  Two CTAs per SM leave
// 128 registers, of which the forms with A in rows spill 20 to 72 bytes.
constexpr int kSgBk = 32, kSgRow = kSgBk + 4, kSgCol = 128 + 4;  // row strides: 16-byte rows, 4 banks apart
constexpr int kSgOp = 128 * kSgRow;                              // floats of one operand's buffer (either layout)
static_assert(kSgBk * kSgCol <= kSgOp && 128 * kSgCol <= 4 * kSgOp, "column layout and the output tile fit");
constexpr int kSgSmem = 4 * kSgOp * int(sizeof(float));

template <int LAYOUT>
__device__ __forceinline__ void sg_stage(const float* X, int ld, int rows, int k0, int K, bool vec, float* sh, int tid) {
  const uint32_t s0 = smem_u32(sh);
  if (vec) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = tid + 256 * u;
      const int r = LAYOUT == kRow ? e >> 3 : 4 * (e & 31), k = LAYOUT == kRow ? 4 * (e & 7) : e >> 5;
      const int left = LAYOUT == kRow ? (r < rows ? K - k0 - k : 0) : (k0 + k < K ? rows - r : 0);
      const int bytes = 4 * max(0, min(4, left));
      const float* src = LAYOUT == kRow ? X + int64_t(r) * ld + k0 + k : X + int64_t(k0 + k) * ld + r;
      cp_async16(s0 + 4 * (LAYOUT == kRow ? r * kSgRow + k : k * kSgCol + r), bytes ? src : X, bytes);
    }
  } else {
#pragma unroll 4
    for (int u = 0; u < 16; ++u) {
      const int e = tid + 256 * u;
      const int r = LAYOUT == kRow ? e >> 5 : e & 127, k = LAYOUT == kRow ? e & 31 : e >> 7;
      const bool ok = r < rows && k0 + k < K;
      const float* src = LAYOUT == kRow ? X + int64_t(r) * ld + k0 + k : X + int64_t(k0 + k) * ld + r;
      cp_async4(s0 + 4 * (LAYOUT == kRow ? r * kSgRow + k : k * kSgCol + r), ok ? src : X, ok ? 4 : 0);
    }
  }
}
// index of entry q (of 8) along an operand's rows for position `p` of P in the warp
template <int LAYOUT, int P>
__device__ __forceinline__ int sg_row(int p, int q) { return LAYOUT == kRow ? p + P * q : 8 * p + q; }
// k values kk, kk + 1 of the thread's eight rows
template <int LAYOUT, int P>
__device__ __forceinline__ void sg_frag(const float* sh, int base, int p, int kk, float (&f)[2][8]) {
  if (LAYOUT == kRow) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float2 v = *reinterpret_cast<const float2*>(sh + (base + p + P * q) * kSgRow + kk);
      f[0][q] = v.x;
      f[1][q] = v.y;
    }
  } else {
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<float4*>(&f[e][4 * h]) =
            *reinterpret_cast<const float4*>(sh + (kk + e) * kSgCol + base + 8 * p + 4 * h);
  }
}

template <int MODE, int AL, int BL>
__global__ void __launch_bounds__(256, 2) gemm32_kernel(const GemmTask* __restrict__ tasks, const float* Ab,
                                                        const float* Bb, float* Cb) {
  extern __shared__ __align__(16) float sgm[];
  const GemmTask tk = tasks[blockIdx.x];
  const float* A = Ab + tk.a;
  const float* B = Bb + tk.b;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wr = 32 * (warp & 3), wc = 64 * (warp >> 2), ly = lane >> 3, lx = lane & 7;
  const bool avec = ((reinterpret_cast<uintptr_t>(A) & 15) == 0) && (tk.lda & 3) == 0;
  const bool bvec = ((reinterpret_cast<uintptr_t>(B) & 15) == 0) && (tk.ldb & 3) == 0;
  const bool active = wr < tk.m && wc < tk.n;
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  const int nk = (tk.k + kSgBk - 1) / kSgBk;
  auto stage = [&](int t) {
    float* buf = sgm + (t & 1) * 2 * kSgOp;
    sg_stage<AL>(A, tk.lda, tk.m, t * kSgBk, tk.k, avec, buf, tid);
    sg_stage<BL>(B, tk.ldb, tk.n, t * kSgBk, tk.k, bvec, buf + kSgOp, tid);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  chain_wait();
  stage(0);
  if (MODE == kSub || MODE == kAdd) prefetch_c<128, 256>(Cb + tk.c, tk.ldc, tk.m, tk.n, tid);
  for (int t = 0; t < nk; ++t) {
    if (t + 1 < nk) {
      stage(t + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    if (active) {
      const float* As = sgm + (t & 1) * 2 * kSgOp;
      const float* Bs = As + kSgOp;
      const int kn = min(kSgBk, (tk.k - t * kSgBk + 1) & ~1);
#pragma unroll 4
      for (int kk = 0; kk < kn; kk += 2) {
        float a[2][8], b[2][8];
        sg_frag<AL, 4>(As, wr, ly, kk, a);
        sg_frag<BL, 8>(Bs, wc, lx, kk, b);
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[e][i], b[e][j], acc[i][j]);
      }
    }
    __syncthreads();
  }
  chain_trigger();
  // through shared memory, so that whole rows of C are read and written
  float* tile = sgm;
  if (active) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float* row = tile + (wr + sg_row<AL, 4>(ly, i)) * kSgCol + wc;
      if (BL == kRow) {
#pragma unroll
        for (int j = 0; j < 8; ++j) row[lx + 8 * j] = acc[i][j];
      } else {
        *reinterpret_cast<float4*>(row + 8 * lx) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        *reinterpret_cast<float4*>(row + 8 * lx + 4) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
      }
    }
  }
  __syncthreads();
  rows_to_global<MODE, 128, 8>(tile, kSgCol, Cb + tk.c, tk.ldc, tk.m, tk.n, warp, lane);
}

template <typename T, int MODE, int AL, int BL>
static void gemm_layout(const GemmTask* t, int n, const T* A, const T* B, T* C, cudaStream_t st) {
  if constexpr (sizeof(T) == sizeof(float)) {
    allow_smem<gemm32_kernel<MODE, AL, BL>>(kSgSmem);
    launch_chained(gemm32_kernel<MODE, AL, BL>, n, 256, kSgSmem, st, t, A, B, C);
  } else {
    launch_chained(gemm64_kernel<MODE, AL, BL>, n, 256, 0, st, t, A, B, C);
  }
}

template <typename T, int MODE>
static void gemm_mode(const GemmTask* t, int n, const T* A, const T* B, T* C, int al, int bl, cudaStream_t st) {
  if (al == kRow && bl == kRow) gemm_layout<T, MODE, kRow, kRow>(t, n, A, B, C, st);
  else if (al == kRow && bl == kCol) gemm_layout<T, MODE, kRow, kCol>(t, n, A, B, C, st);
  else if (al == kCol && bl == kRow) gemm_layout<T, MODE, kCol, kRow>(t, n, A, B, C, st);
  else gemm_layout<T, MODE, kCol, kCol>(t, n, A, B, C, st);
}

// ------------------------------------------------------------ narrow GEMM
// Products with at most 8 output columns (solves with few right-hand sides) are
// bandwidth work: one CTA per task (m <= 128 rows) streams its A once,
// coalesced, against B staged in shared memory.  Each thread keeps 16 to 32
// independent loads in flight, and the CTA holds only 8 KB of shared memory
// (FP32), so that it fits on an SM beside a resident tensor-core CTA.  NB (1 or
// 8) bounds the task's columns.  Every CTA reads all of its A and B before it
// writes C (in-place solves stay valid).
constexpr int kNarrowN = 8;
constexpr int kNarrowBEnt = 2048;  // shared entries: staged B (NB x k chunk), then the k-split partial sums
// Column layout: loads in flight per thread.  Measured over the 54 launches of a 301 x 203
// evaluation with four right-hand sides: with 8, and a chunk's last ones one at a time,
// 1,468 us; 8 in every round 796; 16 697 (the evaluation: 5.29, 4.77, 4.68 ms; 32 4.73).
constexpr int kNarrowRows = 16;

// Sum of v[r] over the 32 lanes of the warp for the eight rows r: lanes with
// (lane >> 2) == r receive row r (a butterfly that halves the rows each lane
// carries at every step: 9 shuffles instead of 8 x 5).
template <typename T>
__device__ __forceinline__ T warp_sum8(const T (&v)[8], int lane) {
  const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
  T w[4], x[2];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const T send = b4 ? v[r] : v[r + 4], keep = b4 ? v[r + 4] : v[r];
    w[r] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const T send = b3 ? w[r] : w[r + 2], keep = b3 ? w[r + 2] : w[r];
    x[r] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  T y = (b2 ? x[1] : x[0]) + __shfl_xor_sync(0xffffffffu, b2 ? x[0] : x[1], 4);
  y += __shfl_xor_sync(0xffffffffu, y, 2);
  y += __shfl_xor_sync(0xffffffffu, y, 1);
  return y;
}

template <int MODE, typename T>
__device__ __forceinline__ void narrow_store(T* dst, T v) {
  if (MODE == kSub) *dst -= v;
  else if (MODE == kStore) *dst = v;
  else if (MODE == kNegStore) *dst = -v;
  else *dst += v;
}

template <typename T, int MODE, int AL, int NB>
__global__ void __launch_bounds__(256) gemv_kernel(const GemmTask* __restrict__ tasks, const T* Ab, const T* Bb,
                                                   T* Cb, int bl) {
  constexpr int kc = kNarrowBEnt / NB;  // k values per staged chunk (a multiple of 64)
  __shared__ T sh[kNarrowBEnt];         // Bs[j * kc + kk] while streaming, partial sums after
  const GemmTask tk = tasks[blockIdx.x];
  const T* A = Ab + tk.a;
  const T* B = Bb + tk.b;
  T* C = Cb + tk.c;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = tk.n, m = tk.m;
  chain_wait();
  if (AL == kRow) {
    // rows in batches of 8; warp w owns batches w and w + 8 (m <= 128); lanes
    // stride along k, 64 k values per step
    constexpr int BAT = NB == 1 ? 2 : 1;  // batches loaded together
    T res[2][NB];
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int j = 0; j < NB; ++j) res[q][j] = T(0);
    for (int k0 = 0; k0 < tk.k; k0 += kc) {
      const int kn = min(kc, tk.k - k0);
      const int kp = (kn + 63) & ~63;
      __syncthreads();
      for (int e = tid; e < kp * NB; e += 256) {
        const int j = e / kp, kk = e - j * kp;
        T v = T(0);
        if (kk < kn && j < n) v = bl == kRow ? B[int64_t(j) * tk.ldb + k0 + kk] : B[int64_t(k0 + kk) * tk.ldb + j];
        sh[j * kc + kk] = v;
      }
      __syncthreads();
#pragma unroll
      for (int b0 = 0; b0 < 2; b0 += BAT) {
        if (8 * (warp + 8 * b0) >= m) break;
        T v[BAT][8][NB];
#pragma unroll
        for (int q = 0; q < BAT; ++q)
#pragma unroll
          for (int r = 0; r < 8; ++r)
#pragma unroll
            for (int j = 0; j < NB; ++j) v[q][r][j] = T(0);
        for (int kk0 = 0; kk0 < kn; kk0 += 64) {
          T a[BAT][8][2];
#pragma unroll
          for (int q = 0; q < BAT; ++q)
#pragma unroll
            for (int r = 0; r < 8; ++r) {
              const int i = 8 * (warp + 8 * (b0 + q)) + r;
              const T* ar = A + int64_t(i) * tk.lda + k0 + kk0 + lane;
#pragma unroll
              for (int u = 0; u < 2; ++u)
                a[q][r][u] = (i < m && kk0 + lane + 32 * u < kn) ? ar[32 * u] : T(0);
            }
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            T bv[NB];
#pragma unroll
            for (int j = 0; j < NB; ++j) bv[j] = sh[j * kc + kk0 + lane + 32 * u];
#pragma unroll
            for (int q = 0; q < BAT; ++q)
#pragma unroll
              for (int r = 0; r < 8; ++r)
#pragma unroll
                for (int j = 0; j < NB; ++j) v[q][r][j] = fma(a[q][r][u], bv[j], v[q][r][j]);
          }
        }
#pragma unroll
        for (int q = 0; q < BAT; ++q)
#pragma unroll
          for (int j = 0; j < NB; ++j) {
            T col[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) col[r] = v[q][r][j];
            res[b0 + q][j] += warp_sum8(col, lane);
          }
      }
    }
    __syncthreads();
    if ((lane & 3) == 0) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int i = 8 * (warp + 8 * q) + (lane >> 2);
        if (i < m) {
#pragma unroll
          for (int j = 0; j < NB; ++j)
            if (j < n) narrow_store<MODE>(C + int64_t(i) * tk.ldc + j, res[q][j]);
        }
      }
    }
  } else {
    // thread (h, i): row i, every H-th k value starting at h; kNarrowRows loads in flight, also
    // in the last ones of a chunk (past it a load repeats its last value and is dropped)
    const int rsh = m <= 32 ? 5 : (m <= 64 ? 6 : 7);
    const int i = tid & ((1 << rsh) - 1), h = tid >> rsh, H = 256 >> rsh;
    T s[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) s[j] = T(0);
    for (int k0 = 0; k0 < tk.k; k0 += kc) {
      const int kn = min(kc, tk.k - k0);
      __syncthreads();
      for (int e = tid; e < kn * NB; e += 256) {
        const int j = e / kn, kk = e - j * kn;
        T v = T(0);
        if (j < n) v = bl == kRow ? B[int64_t(j) * tk.ldb + k0 + kk] : B[int64_t(k0 + kk) * tk.ldb + j];
        sh[j * kc + kk] = v;
      }
      __syncthreads();
      if (i < m) {
        const T* ac = A + int64_t(k0) * tk.lda + i;
        for (int kk = h; kk < kn; kk += kNarrowRows * H) {
          T a[kNarrowRows];
#pragma unroll
          for (int u = 0; u < kNarrowRows; ++u) a[u] = ac[int64_t(min(kk + u * H, kn - 1)) * tk.lda];
#pragma unroll
          for (int u = 0; u < kNarrowRows; ++u)
            if (kk + u * H < kn)
#pragma unroll
              for (int j = 0; j < NB; ++j) s[j] = fma(a[u], sh[j * kc + kk + u * H], s[j]);
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NB; ++j) sh[j * 256 + tid] = s[j];
    __syncthreads();
    for (int e = tid; e < m * n; e += 256) {
      const int ii = e / n, j = e - ii * n;
      T v = T(0);
      for (int hh = 0; hh < H; ++hh) v += sh[j * 256 + (hh << rsh) + ii];
      narrow_store<MODE>(C + int64_t(ii) * tk.ldc + j, v);
    }
  }
}

// ------------------------------------------------------ panel solve (FP32)
// X = A Linv^T for one 64-column diagonal block: tasks with m <= 128 rows,
// n <= 64 columns and k <= 64, both operands in row layout.  A CTA takes ROWS rows
// of a task; it stages them and the block inverse in shared memory as they lie (no
// K loop, one 16-byte load per four values where the rows are aligned), then
// thread (ty, tx) computes the entries (ty + 16 r, tx + 16 c), reading both
// operands four k values at a time without bank conflicts.  A may alias C
// (in-place panel solve; the rows of a task's CTAs are their own): every read
// happens before the first write.  Bound: latency, the launch being one of a
// serial chain per 64 columns.
constexpr int kPanelLd = 68;  // row stride of the staged tiles: 16-byte rows, 4 banks apart
constexpr int panel_smem(int rows) { return (rows + 64) * kPanelLd * int(sizeof(float)); }

// rows x 64 values of X (zero outside m x k) into shared memory, NT threads
template <int ROWS>
__device__ __forceinline__ void panel_stage(const float* X, int ldx, int m, int k, float* sh, int tid) {
  const bool vec = ((reinterpret_cast<uintptr_t>(X) & 15) == 0) && (ldx & 3) == 0;
  float4 v[ROWS / 16];
#pragma unroll
  for (int u = 0; u < ROWS / 16; ++u) {
    const int i = (tid >> 4) + 16 * u, c = 4 * (tid & 15);
    v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < m) {
      const float* x = X + int64_t(i) * ldx + c;
      if (vec && c + 4 <= k) {
        v[u] = *reinterpret_cast<const float4*>(x);
      } else {
        if (c + 0 < k) v[u].x = x[0];
        if (c + 1 < k) v[u].y = x[1];
        if (c + 2 < k) v[u].z = x[2];
        if (c + 3 < k) v[u].w = x[3];
      }
    }
  }
#pragma unroll
  for (int u = 0; u < ROWS / 16; ++u)
    *reinterpret_cast<float4*>(sh + ((tid >> 4) + 16 * u) * kPanelLd + 4 * (tid & 15)) = v[u];
}

template <int MODE, int ROWS>
__global__ void __launch_bounds__(256) panel64_kernel(const GemmTask* __restrict__ tasks, const float* Ab,
                                                      const float* Bb, float* Cb) {
  extern __shared__ __align__(16) float psm[];
  constexpr int kSplit = 128 / ROWS, R = ROWS / 16;
  float* As = psm;                     // As[i * kPanelLd + k] = A(i, k)
  float* Bs = psm + ROWS * kPanelLd;   // Bs[j * kPanelLd + k] = B(j, k)
  const GemmTask tk = tasks[blockIdx.x / kSplit];
  const int row0 = int(blockIdx.x % kSplit) * ROWS, m = min(ROWS, tk.m - row0);
  chain_wait();
  if (m <= 0) return;
  float* C = Cb + tk.c + int64_t(row0) * tk.ldc;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  panel_stage<ROWS>(Ab + tk.a + int64_t(row0) * tk.lda, tk.lda, m, tk.k, As, tid);
  panel_stage<64>(Bb + tk.b, tk.ldb, tk.n, tk.k, Bs, tid);
  float old[R][4];
  if (MODE == kSub || MODE == kAdd) {  // in flight with the operands
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int i = ty + 16 * r, j = tx + 16 * c;
        old[r][c] = (i < m && j < tk.n) ? C[int64_t(i) * tk.ldc + j] : 0.f;
      }
  }
  __syncthreads();
  float acc[R][4];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
#pragma unroll 2
  for (int kk = 0; kk < tk.k; kk += 4) {
    float4 a[R], b[4];
#pragma unroll
    for (int r = 0; r < R; ++r) a[r] = *reinterpret_cast<const float4*>(As + (ty + 16 * r) * kPanelLd + kk);
#pragma unroll
    for (int c = 0; c < 4; ++c) b[c] = *reinterpret_cast<const float4*>(Bs + (tx + 16 * c) * kPanelLd + kk);
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(a[r].x, b[c].x, acc[r][c]);
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(a[r].y, b[c].y, acc[r][c]);
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(a[r].z, b[c].z, acc[r][c]);
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(a[r].w, b[c].w, acc[r][c]);
  }
  chain_trigger();
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = ty + 16 * r, j = tx + 16 * c;
      if (i >= m || j >= tk.n) continue;
      float* dst = C + int64_t(i) * tk.ldc + j;
      if (MODE == kSub) *dst = old[r][c] - acc[r][c];
      else if (MODE == kStore) *dst = acc[r][c];
      else if (MODE == kNegStore) *dst = -acc[r][c];
      else *dst = old[r][c] + acc[r][c];
    }
}

// Fewer rows per CTA while the launch leaves SMs idle: 32 rows up to 152 tasks, 64 up to 304.
template <int MODE, int ROWS>
static void panel64_rows(const GemmTask* t, int n, const float* A, const float* B, float* C, cudaStream_t st) {
  allow_smem<panel64_kernel<MODE, ROWS>>(panel_smem(ROWS));
  launch_chained(panel64_kernel<MODE, ROWS>, n * (128 / ROWS), 256, panel_smem(ROWS), st, t, A, B, C);
}
template <int MODE>
static void panel64_launch(const GemmTask* t, int n, const float* A, const float* B, float* C, cudaStream_t st) {
  if (n <= 152) panel64_rows<MODE, 32>(t, n, A, B, C, st);
  else if (n <= 304) panel64_rows<MODE, 64>(t, n, A, B, C, st);
  else panel64_rows<MODE, 128>(t, n, A, B, C, st);
}

template <typename T, int MODE>
static void gemv_mode(const GemmTask* t, int n, const T* A, const T* B, T* C, int al, int bl, cudaStream_t st,
                      int nmax) {
  if (nmax == 1) {
    if (al == kRow) launch_chained(gemv_kernel<T, MODE, kRow, 1>, n, 256, 0, st, t, A, B, C, bl);
    else launch_chained(gemv_kernel<T, MODE, kCol, 1>, n, 256, 0, st, t, A, B, C, bl);
  } else {
    if (al == kRow) launch_chained(gemv_kernel<T, MODE, kRow, kNarrowN>, n, 256, 0, st, t, A, B, C, bl);
    else launch_chained(gemv_kernel<T, MODE, kCol, kNarrowN>, n, 256, 0, st, t, A, B, C, bl);
  }
}

// The FP32 products run on the tensor cores unless SPDE_TC=0 is set in the environment.
bool tc_gemm_enabled() {
  static int on = -1;
  if (on < 0) {
    const char* e = getenv("SPDE_TC");
    on = (e && e[0] == '0') ? 0 : 1;
  }
  return on == 1;
}

template <typename T>
void launch_gemm(const GemmTask* tasks, int ntasks, const T* A, const T* B, T* C, int mode, int alayout, int blayout,
                 cudaStream_t st, int path, int nmax, unsigned long long wait_ns) {
  if (ntasks <= 0) return;
  if (path == kPathNarrow) {
    switch (mode) {
      case kSub: gemv_mode<T, kSub>(tasks, ntasks, A, B, C, alayout, blayout, st, nmax); break;
      case kStore: gemv_mode<T, kStore>(tasks, ntasks, A, B, C, alayout, blayout, st, nmax); break;
      case kNegStore: gemv_mode<T, kNegStore>(tasks, ntasks, A, B, C, alayout, blayout, st, nmax); break;
      default: gemv_mode<T, kAdd>(tasks, ntasks, A, B, C, alayout, blayout, st, nmax); break;
    }
    return;
  }
  if constexpr (sizeof(T) == sizeof(float)) {
    if (path == kPathPanel && alayout == kRow && blayout == kRow) {
      const float* Af = reinterpret_cast<const float*>(A);
      const float* Bf = reinterpret_cast<const float*>(B);
      float* Cf = reinterpret_cast<float*>(C);
      switch (mode) {
        case kSub: panel64_launch<kSub>(tasks, ntasks, Af, Bf, Cf, st); break;
        case kStore: panel64_launch<kStore>(tasks, ntasks, Af, Bf, Cf, st); break;
        case kNegStore: panel64_launch<kNegStore>(tasks, ntasks, Af, Bf, Cf, st); break;
        default: panel64_launch<kAdd>(tasks, ntasks, Af, Bf, Cf, st); break;
      }
      return;
    }
    if (path == kPathTensor && tc_gemm_enabled()) {
      launch_gemm_tc(tasks, ntasks, reinterpret_cast<const float*>(A), reinterpret_cast<const float*>(B),
                     reinterpret_cast<float*>(C), mode, alayout, blayout, st, wait_ns);
      return;
    }
  }
  switch (mode) {
    case kSub: gemm_mode<T, kSub>(tasks, ntasks, A, B, C, alayout, blayout, st); break;
    case kStore: gemm_mode<T, kStore>(tasks, ntasks, A, B, C, alayout, blayout, st); break;
    case kNegStore: gemm_mode<T, kNegStore>(tasks, ntasks, A, B, C, alayout, blayout, st); break;
    default: gemm_mode<T, kAdd>(tasks, ntasks, A, B, C, alayout, blayout, st); break;
  }
}

template void launch_gemm<double>(const GemmTask*, int, const double*, const double*, double*, int, int, int,
                                  cudaStream_t, int, int, unsigned long long);
template void launch_gemm<float>(const GemmTask*, int, const float*, const float*, float*, int, int, int,
                                 cudaStream_t, int, int, unsigned long long);

// ------------------------------------------------------------ diagonal blocks
// The mixed plan's diagonal blocks are eliminated in double-float arithmetic (value =
// hi + lo, two FP32 numbers, about 44 significant bits; Dekker/Knuth error-free
// transformations with FMA), which runs on the FP32 pipe instead of the narrow FP64
// one (an FP32 sweep measured 1e-6 relative log-likelihood error against 1e-7 at 960k
// nodes).  Pivots are converted to FP64 for the log-determinant; L and L^-1 are
// rounded to FP32 for storage (L^-1 from the FP32 L).
constexpr int kMaxNbk = 64;

struct DF {
  float hi, lo;
};
// The _rn intrinsics keep the compiler from contracting the error-free
// transformations into FMAs.
__device__ __forceinline__ DF df_renorm(float s, float e) {
  const float h = __fadd_rn(s, e);
  return DF{h, __fsub_rn(e, __fsub_rn(h, s))};
}
// b * c
__device__ __forceinline__ DF df_mul(DF b, DF c) {
  const float p = __fmul_rn(b.hi, c.hi);
  float e = fmaf(b.hi, c.hi, -p);
  e = fmaf(b.hi, c.lo, e);
  e = fmaf(b.lo, c.hi, e);
  return df_renorm(p, e);
}
// a - b * c
__device__ __forceinline__ DF df_fms(DF a, DF b, DF c) {
  const float p = __fmul_rn(b.hi, c.hi);
  float e = fmaf(b.hi, c.hi, -p);
  e = fmaf(b.hi, c.lo, e);
  e = fmaf(b.lo, c.hi, e);
  const float s = __fsub_rn(a.hi, p);
  const float v = __fsub_rn(s, a.hi);
  float err = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, v)), __fsub_rn(-p, v));
  err = __fadd_rn(err, __fsub_rn(a.lo, e));
  return df_renorm(s, err);
}
// Two FP32 values per register pair and instruction (add, mul and fma.rn.f32x2: each
// half rounds as the scalar instruction does)
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2_pack(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 f2_unpack(F2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
  return r;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
struct DF2 {
  F2 hi, lo;
};
// df_fms for two entries: x - s a, the same roundings in the same order; ns = -s.hi,
// and a difference u - w is formed as fma(w, -1, u), which rounds once like it
__device__ __forceinline__ DF2 df2_fms(DF2 x, DF2 s, F2 ns, DF2 a, F2 minus1) {
  const F2 np = f2_mul(ns, a.hi);  // -p
  F2 e = f2_fma(s.hi, a.hi, np);
  e = f2_fma(s.hi, a.lo, e);
  e = f2_fma(s.lo, a.hi, e);
  const F2 h = f2_add(x.hi, np);
  const F2 v = f2_fma(x.hi, minus1, h);
  F2 t = f2_fma(f2_fma(v, minus1, h), minus1, x.hi);  // x.hi - (h - v)
  t = f2_add(t, f2_fma(v, minus1, np));
  t = f2_add(t, f2_fma(e, minus1, x.lo));
  const F2 r = f2_add(h, t);
  return DF2{r, f2_fma(f2_fma(h, minus1, r), minus1, t)};
}
// 1 / d: FP32 reciprocal estimate refined by one Newton step with a
// double-float residual (the step squares the estimate's relative error, so
// the hardware approximation is enough)
__device__ __forceinline__ DF df_rcp(DF d) {
  const float r = __fdividef(1.0f, d.hi);
  const DF one_minus = df_fms(DF{1.0f, 0.0f}, d, DF{r, 0.0f});  // 1 - d r
  return df_renorm(r, __fmul_rn(r, one_minus.hi));
}

// 1 / sqrt(d) rounded to FP32 for a double-float pivot, without the (narrow)
// FP64 pipe: the hardware estimate y refined by one Newton-Raphson step
// y + y e / 2 with the residual e = 1 - d y^2 formed from the exact square of y
// (FMA error terms), which leaves an error far below FP32 rounding.
__device__ __forceinline__ float df_rsqrt(DF d) {
  const float y = rsqrtf(d.hi);
  const float p = __fmul_rn(y, y);
  const float pe = fmaf(y, y, -p);        // y^2 = p + pe exactly
  float e = fmaf(-d.hi, p, 1.0f);         // 1 - d_hi p, one rounding
  e = fmaf(-d.hi, pe, e);
  e = fmaf(-d.lo, p, e);
  return fmaf(0.5f * y, e, y);
}

// Factorisation of one diagonal block A = L L^T (w <= 64) and its inverse, one CTA per
// block; T the storage type, the elimination in double-float (FP32 storage) or FP64.
//
// The elimination is written A_ik -= (a_ic / d_c) a_kc, so that the pivots d_c
// and the columns a_ic (at the time column c is eliminated) stay in the elimination's
// arithmetic and L_ic = a_ic / sqrt(d_c) is rounded to storage once, at the end.  Every entry
// takes its updates in the order of c, so the result does not depend on how the
// work is split over threads.
//
// Bound: latency.  The blocks of a front's top levels are a serial chain with
// one block per launch, so the kernel is built around the chain from pivot to
// pivot.  It goes by 16-column panels.  A panel is eliminated by one warp per 16
// rows below its diagonal block: lanes 0-15 hold the diagonal block's rows (the
// same in every warp), lanes 16-31 the warp's own rows, one row per lane in
// registers, so that pivots and multipliers travel by shuffle and no warp waits for
// another inside a panel.  Between the two barriers around a panel a warp writes only
// rows that no other warp reads there: its own rows in place, and the diagonal block's,
// which every warp loads, into the same rows of the other panel buffer, where the next
// panel writes only rows below them.  The trailing rank-16 update is spread over all 256
// threads, each holding the entries (ty + 16 m, tx + 16 n), n <= m, in registers.
// Then L^-1 (FP32) by 16-column sub-blocks: the four diagonal inverses (a warp
// each, one lane per column, right-looking so that the partial sums of all rows
// advance together) beside the pivot logarithms on a fifth warp, then the
// off-diagonal blocks by distance from the diagonal, X_ij = -X_ii (sum_{i > k >= j}
// L_ik X_kj), the factor's entries read four at a time.
// The double-float updates (14 FP32 operations each) issue in pairs of entries as
// add, mul and fma.f32x2, half the instructions of a panel's and a trailing update's
// chain.  Measured at 100 x 100 x 24 (mean over its launches, mostly of one to a few
// blocks): 31.4 us, with scalar operations 36.7; the columns exchanged through shared
// memory and the inverse by rows, without pairs, took 67 us for one block.  Two CTAs
// per SM: with three the registers spill the pairs (32.2 us), and the levels with
// many blocks gain nothing from the third (100 x 100 x 24 evaluation 66.4 ms both).
// The inverse finished by idle warps during the next panel was slower (39.8 us).
constexpr int kDfSub = 16;
constexpr int kDfLd = kMaxNbk + 4;          // row stride of L and L^-1 in shared memory (16-byte rows)
constexpr int kDfPan = kDfSub + 2;          // row stride of a panel in shared memory
template <typename T>
constexpr int potrf_smem() { return (2 * kMaxNbk * kDfLd + 3 * kDfSub * kDfSub) * int(sizeof(T)); }

// The elimination's arithmetic by storage type: numbers, their shared-memory form,
// products, reciprocal and square root of a pivot.
template <typename T>
struct Elim;
template <>
struct Elim<float> {
  using Num = DF;
  using Pair = float2;  // in shared memory
  static constexpr int kMinCtas = 2;
  static __device__ __forceinline__ DF from(float v) { return DF{v, 0.0f}; }
  static __device__ __forceinline__ DF load(Pair v) { return DF{v.x, v.y}; }
  static __device__ __forceinline__ Pair pack(DF v) { return make_float2(v.hi, v.lo); }
  static __device__ __forceinline__ DF shfl(DF v, int lane) {
    return DF{__shfl_sync(0xffffffffu, v.hi, lane), __shfl_sync(0xffffffffu, v.lo, lane)};
  }
  static __device__ __forceinline__ DF mul(DF a, DF b) { return df_mul(a, b); }
  static __device__ __forceinline__ DF fms(DF a, DF b, DF c) { return df_fms(a, b, c); }
  // two entries at once: x0 -= s0 a0, x1 -= s1 a1
  static __device__ __forceinline__ void fms2(DF& x0, DF& x1, DF s0, DF s1, DF a0, DF a1) {
    const DF2 x = df2_fms(DF2{f2_pack(x0.hi, x1.hi), f2_pack(x0.lo, x1.lo)},
                          DF2{f2_pack(s0.hi, s1.hi), f2_pack(s0.lo, s1.lo)}, f2_pack(-s0.hi, -s1.hi),
                          DF2{f2_pack(a0.hi, a1.hi), f2_pack(a0.lo, a1.lo)}, f2_pack(-1.0f, -1.0f));
    const float2 h = f2_unpack(x.hi), l = f2_unpack(x.lo);
    x0 = DF{h.x, l.x};
    x1 = DF{h.y, l.y};
  }
  static __device__ __forceinline__ DF rcp(DF d) { return df_rcp(d); }
  // of a pivot: what `root` holds, and from it 1 / sqrt(d), sqrt(d) and an entry of L
  static __device__ __forceinline__ float root(DF d) { return df_rsqrt(d); }
  static __device__ __forceinline__ float inv(float r) { return r; }
  static __device__ __forceinline__ float diag(float r) { return 1.0f / r; }
  static __device__ __forceinline__ float entry(DF v, float r) { return (v.hi + v.lo) * r; }
  static __device__ __forceinline__ bool bad(DF d) { return !(d.hi > 0.0f) || !isfinite(d.hi); }
  static __device__ __forceinline__ double wide(DF v) { return double(v.hi) + double(v.lo); }
};
template <>
struct Elim<double> {
  using Num = double;
  using Pair = double;
  static constexpr int kMinCtas = 2;
  static __device__ __forceinline__ double from(double v) { return v; }
  static __device__ __forceinline__ double load(Pair v) { return v; }
  static __device__ __forceinline__ Pair pack(double v) { return v; }
  static __device__ __forceinline__ double shfl(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }
  static __device__ __forceinline__ double mul(double a, double b) { return a * b; }
  static __device__ __forceinline__ double fms(double a, double b, double c) { return fma(-b, c, a); }
  static __device__ __forceinline__ void fms2(double& x0, double& x1, double s0, double s1, double a0, double a1) {
    x0 = fma(-s0, a0, x0);
    x1 = fma(-s1, a1, x1);
  }
  // 1 / d for d > 0: the FP32 reciprocal of the significand and two Newton steps
  // (four FP64 operations instead of a full division on the narrow pipe); pivots
  // outside the normal range of d and 1 / d take the division.  The steps leave 2^-88 before the
  // last rounding: 4 10^8 random significands, with estimates up to two units off, all gave the
  // division's result
  static __device__ __forceinline__ double rcp(double d) {
    const long long b = __double_as_longlong(d);
    const int f = int(b >> 52);
    if (f < 2 || f > 2044) return 1.0 / d;
    const double m = __longlong_as_double((b & 0xFFFFFFFFFFFFFll) | (1023ll << 52));  // in [1, 2)
    double y = double(__fdividef(1.0f, float(m)));
    y = fma(y, fma(-m, y, 1.0), y);
    y = fma(y, fma(-m, y, 1.0), y);
    return __longlong_as_double(__double_as_longlong(y) - (static_cast<long long>(f - 1023) << 52));
  }
  // the root itself, so that L takes one division (rsqrt is not correctly rounded, and a
  // product with it rounds again)
  static __device__ __forceinline__ double root(double d) { return sqrt(d); }
  static __device__ __forceinline__ double inv(double r) { return 1.0 / r; }
  static __device__ __forceinline__ double diag(double r) { return r; }
  static __device__ __forceinline__ double entry(double v, double r) { return v / r; }
  static __device__ __forceinline__ bool bad(double d) { return !(d > 0.0) || !isfinite(d); }
  static __device__ __forceinline__ double wide(double v) { return v; }
};

__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
  *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(p);
}
__device__ __forceinline__ void load4(const double* p, double (&v)[4]) {
  *reinterpret_cast<double2*>(v) = *reinterpret_cast<const double2*>(p);
  *reinterpret_cast<double2*>(v + 2) = *reinterpret_cast<const double2*>(p + 2);
}

template <typename T>
__global__ void __launch_bounds__(256, Elim<T>::kMinCtas)
    potrf_kernel(const DiagTask* __restrict__ tasks, T* L, T* dinv,
                 double* logpiv, int* err) {
  using E = Elim<T>;
  using Num = typename E::Num;
  using Pair = typename E::Pair;
  // L and L^-1; before that, two panel buffers and the panel's multipliers
  extern __shared__ __align__(16) uint8_t potrf_sm[];
  __shared__ Pair dp[kMaxNbk];
  __shared__ T root[kMaxNbk], rinv[kMaxNbk];
  __shared__ int bad;
  static_assert(2 * kMaxNbk * kDfLd * sizeof(T) >= 3 * kMaxNbk * kDfPan * sizeof(Pair), "panel buffers fit");
  T (*Ls)[kDfLd] = reinterpret_cast<T (*)[kDfLd]>(potrf_sm);
  T (*Xs)[kDfLd] = Ls + kMaxNbk;
  T* Tb = &Xs[kMaxNbk][0];                     // 3 x 256 products of the inverse
  Pair (*pan0)[kDfPan] = reinterpret_cast<Pair (*)[kDfPan]>(potrf_sm);
  Pair (*mul)[kDfPan] = pan0 + 2 * kMaxNbk;    // S_ic = a_ic / d_c
  const DiagTask tk = tasks[blockIdx.x];
  const int w = tk.w;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ty = tid >> 4, tx = tid & 15;
  T* blk = L + tk.a;
  chain_wait();
  Num r[4][4];                               // n <= m used
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n <= m; ++n) {
      const int i = ty + 16 * m, k = tx + 16 * n;
      r[m][n] = E::from((k <= i && i < w) ? blk[int64_t(i) * tk.lda + k] : T(0));
    }
  if (tid == 0) bad = 0;
  for (int jb = 0; 16 * jb < w; ++jb) {
    Pair (*pan)[kDfPan] = pan0 + (jb & 1) * kMaxNbk;
    Pair (*fin)[kDfPan] = pan0 + (~jb & 1) * kMaxNbk;  // takes the panel's finished diagonal rows
    const int c0 = 16 * jb, cw = min(kDfSub, w - c0);
    // block column jb to shared memory (the register indices are compile-time constants)
#pragma unroll
    for (int n = 0; n < 4; ++n)
      if (n == jb) {
#pragma unroll
        for (int m = n; m < 4; ++m) pan[ty + 16 * m][tx] = E::pack(r[m][n]);
      }
    __syncthreads();
    if (warp == 0 || c0 + 16 * (warp + 1) < w) {
      const int row = lane < 16 ? c0 + lane : min(c0 + 16 * (warp + 1) + lane - 16, kMaxNbk - 1);
      Num x[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) x[k] = E::load(pan[row][k]);
      __syncwarp();
      const bool own = lane >= 16 ? c0 + 16 * (warp + 1) < w : warp == 0;  // this lane's row is written by this warp
      Num piv = E::from(T(1));
      bool failed = false;
      // columns >= cw are zero: their pivot counts as 1 and they change nothing
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        Num d = E::shfl(x[j], j);
        const bool nonpos = E::bad(d);
        if (nonpos) d = E::from(T(1));
        const Num sj = E::mul(x[j], E::rcp(d));
        if (lane == j) piv = d;
        failed |= nonpos && j < cw;
        if (own) {
          (lane < 16 ? fin : pan)[row][j] = E::pack(x[j]);
          mul[row][j] = E::pack(sj);
        }
        if (j % 2 == 0 && j < 15) x[j + 1] = E::fms(x[j + 1], sj, E::shfl(x[j], j + 1));
#pragma unroll
        for (int k = (j + 2) & ~1; k < 16; k += 2)
          E::fms2(x[k], x[k + 1], sj, sj, E::shfl(x[j], k), E::shfl(x[j], k + 1));
      }
      if (warp == 0 && lane < cw) {
        dp[c0 + lane] = E::pack(piv);
        if (failed) bad = 1;
      }
    }
    __syncthreads();
    auto trailing = [&](auto block) {
      constexpr int n = decltype(block)::value;
#pragma unroll
      for (int m = n; m < 4; ++m) {  // the panel's final entries
        r[m][n] = E::load((m == n ? fin : pan)[ty + 16 * m][tx]);
      }
      if (c0 + 16 < w) {
#pragma unroll 4
        for (int c = 0; c < kDfSub; c += 2) {  // two columns per 16-byte load
          Pair sv[4][2], av[4][2];
#pragma unroll
          for (int m = n + 1; m < 4; ++m) {
            *reinterpret_cast<float4*>(sv[m]) = *reinterpret_cast<const float4*>(&mul[ty + 16 * m][c]);
            *reinterpret_cast<float4*>(av[m]) = *reinterpret_cast<const float4*>(&pan[tx + 16 * m][c]);
          }
          auto s_of = [&](int m, int h) { return E::load(sv[m][h]); };
          auto a_of = [&](int q, int h) { return E::load(av[q][h]); };
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (n == 0) {
              E::fms2(r[2][1], r[2][2], s_of(2, h), s_of(2, h), a_of(1, h), a_of(2, h));
              E::fms2(r[3][1], r[3][2], s_of(3, h), s_of(3, h), a_of(1, h), a_of(2, h));
              E::fms2(r[1][1], r[3][3], s_of(1, h), s_of(3, h), a_of(1, h), a_of(3, h));
            } else if (n == 1) {
              E::fms2(r[2][2], r[3][2], s_of(2, h), s_of(3, h), a_of(2, h), a_of(2, h));
              r[3][3] = E::fms(r[3][3], s_of(3, h), a_of(3, h));
            } else if (n == 2) {
              r[3][3] = E::fms(r[3][3], s_of(3, h), a_of(3, h));
            }
          }
        }
      }
    };
    switch (jb) {
      case 0: trailing(IntC<0>{}); break;
      case 1: trailing(IntC<1>{}); break;
      case 2: trailing(IntC<2>{}); break;
      default: trailing(IntC<3>{}); break;
    }
  }
  __syncthreads();
  if (tid < w) {
    root[tid] = E::root(E::load(dp[tid]));
    rinv[tid] = E::inv(root[tid]);
  }
  __syncthreads();
  // L = a_ik / sqrt(d_k), zero above the diagonal
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int i = ty + 16 * m, k = tx + 16 * n;
      if (i < w && k < w) {
        T v = T(0);
        if (n <= m) {
          if (k < i) v = E::entry(r[m][n], root[k]);
          else if (k == i) v = E::diag(root[k]);
        }
        Ls[i][k] = v;
        blk[int64_t(i) * tk.lda + k] = v;
      }
    }
  __syncthreads();
  const int nsb = (w + kDfSub - 1) / kDfSub;
  if (warp < nsb) {
    // diagonal 16 x 16 inverse of sub-block `warp`, lane = column: x_ii = -(sum_{k < ii} L_(ii,k) x_k) / L_(ii,ii)
    if (lane < kDfSub) {
      const int c0 = warp * kDfSub, cw = min(kDfSub, w - c0), c = lane;
      T sum[kDfSub];
#pragma unroll
      for (int ii = 0; ii < kDfSub; ++ii) sum[ii] = T(0);
#pragma unroll
      for (int k = 0; k < kDfSub; ++k) {
        if (k >= cw) break;
        T x = T(0);
        if (k == c) x = rinv[c0 + k];
        else if (k > c) x = -sum[k] * rinv[c0 + k];
        Xs[c0 + k][c0 + c] = x;
#pragma unroll
        for (int ii = k + 1; ii < kDfSub; ++ii)
          if (ii < cw) sum[ii] = fma(Ls[c0 + ii][c0 + k], x, sum[ii]);
      }
    }
  } else if (warp == 7) {
    double s = 0.0;
    for (int j = lane; j < w; j += 32) s += 0.5 * log(E::wide(E::load(dp[j])));
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) {
      logpiv[blockIdx.x] = s;
      if (bad) atomicCAS(err, -1, tk.front);
    }
  }
  __syncthreads();
  // off-diagonal blocks by distance dd: T = sum_k L_(bi,k) X_(k,bj), then X_(bi,bj) = -X_(bi,bi) T
#pragma unroll
  for (int dd = 1; dd < 4; ++dd) {
    if (dd >= nsb) break;
#pragma unroll
    for (int pi = 0; pi < 4 - dd; ++pi) {
      const int i = (dd + pi) * kDfSub + ty;  // rows >= w compute values that nothing reads
      T s = T(0);
#pragma unroll
      for (int k4 = 4 * pi; k4 < 4 * (pi + dd); ++k4) {
        T l[4];
        load4(&Ls[i][4 * k4], l);
#pragma unroll
        for (int e = 0; e < 4; ++e) s = fma(l[e], Xs[4 * k4 + e][pi * kDfSub + tx], s);
      }
      Tb[(pi << 8) + tid] = s;
    }
    __syncthreads();
#pragma unroll
    for (int pi = 0; pi < 4 - dd; ++pi) {
      const int bi = dd + pi, i = bi * kDfSub + ty;
      T s = T(0);
#pragma unroll
      for (int r4 = 0; r4 < kDfSub / 4; ++r4) {
        T xr[4];
        load4(&Xs[i][bi * kDfSub + 4 * r4], xr);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const T nx = fma(xr[e], Tb[(pi << 8) + ((4 * r4 + e) << 4) + tx], s);
          if (4 * r4 + e <= ty) s = nx;
        }
      }
      Xs[i][pi * kDfSub + tx] = -s;
    }
    __syncthreads();
  }
  chain_trigger();
  T* dvp = dinv + tk.dinv;
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int i = ty + 16 * m, c = tx + 16 * n;
      if (i < w && c < w) dvp[int64_t(i) * kMaxNbk + c] = c <= i ? Xs[i][c] : T(0);
    }
}

template <typename T>
void launch_potrf(const DiagTask* tasks, int ntasks, T* L, T* dinv, double* logpiv, int* err, cudaStream_t st) {
  if (ntasks <= 0) return;
  allow_smem<potrf_kernel<T>>(potrf_smem<T>());
  launch_chained(potrf_kernel<T>, ntasks, 256, potrf_smem<T>(), st, tasks, L, dinv, logpiv, err);
}
template void launch_potrf<double>(const DiagTask*, int, double*, double*, double*, int*, cudaStream_t);
template void launch_potrf<float>(const DiagTask*, int, float*, float*, double*, int*, cudaStream_t);

// ------------------------------------------------------------- extend-add
// The lower triangle of a front from its children's update blocks: entry (i, j) takes
// child 0's and child 1's value, in that order, where they have one (src0 / src1 hold,
// for every position of the front, its index in that child's update block or -1).
// Columns inside the separator are added into the front's panel P (which holds Q);
// the others start the front's own update block U, whose unmapped entries become
// zero, so that U is written once and neither cleared nor read.  One warp per row; a
// row is in both children, in one, or in none, which the warp decides once; loads
// are unconditional (an unmapped column reads the child's column 0 and drops it), so
// that a lane's entries overlap.  Bound: memory (4 bytes read per child entry, 4
// written per U entry).  Measured per 100 x 100 x 24 evaluation (two factorisations):
// 3.7 ms, against 5.6 ms for two read-modify-write launches per level and the clearing
// of the update blocks; with a branch per load 6.3 ms, four entries in flight 4.3 ms.
constexpr int kExtUnroll = 8;

// Columns [0, n) of a row; CH: bit 0 child 0 has the row (a0), bit 1 child 1 (a1).
// ADD: dst += the children's values where there are any, else dst = their sum.
template <typename T, int CH, bool ADD>
__device__ __forceinline__ void extend_row(const int* __restrict__ m0, const int* __restrict__ m1,
                                           const T* a0, const T* a1, T* dst, int n, int lane) {
  for (int j0 = lane; j0 < n; j0 += 32 * kExtUnroll) {
    T v0[kExtUnroll], v1[kExtUnroll], o[kExtUnroll];
    int x0[kExtUnroll], x1[kExtUnroll];
#pragma unroll
    for (int u = 0; u < kExtUnroll; ++u) {
      const int j = min(j0 + 32 * u, n - 1);
      x0[u] = (CH & 1) ? m0[j] : -1;
      x1[u] = (CH & 2) ? m1[j] : -1;
      if (ADD) o[u] = dst[j];
    }
#pragma unroll
    for (int u = 0; u < kExtUnroll; ++u) {
      v0[u] = (CH & 1) ? a0[max(x0[u], 0)] : T(0);
      v1[u] = (CH & 2) ? a1[max(x1[u], 0)] : T(0);
    }
#pragma unroll
    for (int u = 0; u < kExtUnroll; ++u) {
      const int j = j0 + 32 * u;
      const bool h0 = (CH & 1) && x0[u] >= 0, h1 = (CH & 2) && x1[u] >= 0;
      T r = ADD ? o[u] : T(0);
      if (h0) r += v0[u];
      if (h1) r += v1[u];
      if (j < n && (!ADD || h0 || h1)) dst[j] = r;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) extend_kernel(const ExtendTask* __restrict__ tasks,
                                                     const DevFront* __restrict__ fronts, const int* __restrict__ src0,
                                                     const int* __restrict__ src1, const T* Uc,
                                                     T* L, T* Up) {
  const ExtendTask tk = tasks[blockIdx.x];
  const DevFront f = fronts[tk.front];
  const int *m0 = src0 + f.i_off, *m1 = src1 + f.i_off;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const T *U0 = Uc, *U1 = Uc;
  int ld0 = 0, ld1 = 0;
  if (f.child[0] >= 0) { U0 += fronts[f.child[0]].u_off; ld0 = fronts[f.child[0]].ldu; }
  if (f.child[1] >= 0) { U1 += fronts[f.child[1]].u_off; ld1 = fronts[f.child[1]].ldu; }
  chain_wait();
  for (int i = tk.r0 + warp; i < tk.r1; i += 8) {
    const int i0 = m0[i], i1 = m1[i];
    const T* a0 = U0 + int64_t(max(i0, 0)) * ld0;  // this row in each child
    const T* a1 = U1 + int64_t(max(i1, 0)) * ld1;
    T* prow = L + f.p_off + int64_t(i) * f.ld;
    const int pn = min(i + 1, f.ns), un = i + 1 - f.ns;
    T* urow = Up + f.u_off + int64_t(un - 1) * f.ldu;
    const int *u0 = m0 + f.ns, *u1 = m1 + f.ns;
    if (i0 >= 0 && i1 >= 0) {
      extend_row<T, 3, true>(m0, m1, a0, a1, prow, pn, lane);
      extend_row<T, 3, false>(u0, u1, a0, a1, urow, un, lane);
    } else if (i0 >= 0) {
      extend_row<T, 1, true>(m0, m1, a0, a1, prow, pn, lane);
      extend_row<T, 1, false>(u0, u1, a0, a1, urow, un, lane);
    } else if (i1 >= 0) {
      extend_row<T, 2, true>(m0, m1, a0, a1, prow, pn, lane);
      extend_row<T, 2, false>(u0, u1, a0, a1, urow, un, lane);
    } else {
      extend_row<T, 0, false>(u0, u1, a0, a1, urow, un, lane);
    }
  }
}

template <typename T>
void launch_extend(const ExtendTask* tasks, int ntasks, const DevFront* fronts, const int* src0, const int* src1,
                   const T* U_child, T* L, T* U_parent, cudaStream_t st) {
  if (ntasks <= 0) return;
  launch_chained(extend_kernel<T>, ntasks, 256, 0, st, tasks, fronts, src0, src1, U_child, L, U_parent);
}
template void launch_extend<double>(const ExtendTask*, int, const DevFront*, const int*, const int*, const double*,
                                    double*, double*, cudaStream_t);
template void launch_extend<float>(const ExtendTask*, int, const DevFront*, const int*, const int*, const float*, float*,
                                   float*, cudaStream_t);

}  // namespace spde
