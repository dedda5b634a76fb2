// Products of the FP64 plan on the tensor cores: C (op)= A B' in FP64 from exact
// products of integer digits (the splitting of K. Ozaki, T. Ogita, S. Oishi, S. M. Rump,
// "Error-free transformations of matrix multiplication by using fast routines of
// matrix multiplication and its applications", Numer. Algorithms 59, 2012).
//
// Split: every operand row is scaled by a power of two (the row's largest magnitude
// below 1) and written as eight signed base-256 digits,
//   x = 2^e sum_s d_s 2^(-7 - 8 s),  |d_s| <= 128,
// rounded to nearest at 2^-64 of the row's scale: entries down to 2^-10 of the row's
// largest keep all 53 bits, smaller ones lose their last.  Digits are exact in bf16.
// Product: digits i of A and j of B with i + j = o <= 7 (36 products) accumulate in
// the tensor core's FP32 accumulator o: all terms are integers, and over 128 values
// of k their sum does not pass 8 * 128 * 2^14 = 2^24, so every accumulator is exact.
// After each 128 values of k the eight accumulators are added into two 64-bit
// integers per output entry, and at the end one conversion rounds
// 2^(ea + eb) sum_o acc_o 2^(-14 - 8 o) to FP64.
// Error of an entry, besides that rounding: 2 * 2^-64 for the operands' digits and
// 7.1 * 2^-64 for the pairs left out (i + j > 7), per value of k and relative to
// (row scale of A) (row scale of B).  FP64 FMAs round each partial sum at 2^-53 of
// itself, so theirs is larger unless the sums stay 2^10 below the scales' product.
// In a factor they do not matter there (|L_i| |L_j| <= sqrt(Q_ii Q_jj), Cholesky's own
// bound); an inverse, whose rows follow the variances along k, was measured: with standard
// deviations over 2^28 its entries' errors, relative to sqrt(Z_ii Z_jj), are 0.5 to 1.1
// times those of FP64 FMAs (seven digits, 2^-56: up to 11 times).
//
// Why: FP64 is a narrow pipe on this part (two FMAs per clock and SM, 1.26 TFLOP/s),
// while 36 bf16 products cost 36 / 2250 of it.  The eighth digit: fit of 30 x 30 x 24
// 15.6 ms (14.8 with seven), 48 x 48 x 24 53.0 ms (49.6).
//
// Split operands lie in memory that the plan's arenas do not use at the time, as the
// shared-memory images the tensor core reads:
// [64-row tile][32-wide k chunk][digit][8-row group][8-wide k core][row][8 x bf16], 4 KB
// per digit, so that a stage is filled by a few bulk copies.  A CTA computes a
// 128 x 64 tile: the eight accumulators take all 512 TMEM columns, and a stage (eight
// digits of 128 x 32 and 64 x 32) 96 KB, two of which fit in shared memory.
// Bound: the tensor core's shared-memory reads (128 + 64 rows per 128 x 64 product); the
// epilogue's 64 bits x 32 sums leave 24 bytes of spills (96 registers, 576 threads).
#include <cuda_runtime.h>
#include <cstdint>

#include "kernels.cuh"
#include "tc_common.cuh"

namespace spde {

namespace {

constexpr int kDigits = kEmuDigits;
constexpr int kBlkBytes = 4096;                       // 64 rows x 32 k of one digit
constexpr int kChunkBytes = kDigits * kBlkBytes;      // ... of all digits
constexpr int kStageA = 2 * kChunkBytes, kStageBytes = 3 * kChunkBytes;
constexpr int kEmuStages = 2;
constexpr int kEmuSmem = kEmuStages * kStageBytes + 1024;
constexpr int kWindow = 4;                            // chunks between two drains (128 values of k)
constexpr int kEpiWarps = 16;
constexpr int kEmuThreads = (kEpiWarps + 2) * 32;     // epilogue warps, loader, MMA issuer
constexpr unsigned long long kEmuWaitNs = 2000000000ull;
constexpr int kFracBits = 8 * kDigits - 1;            // an operand value in units of 2^-kFracBits of its row's scale
constexpr int kLoBits = 8 * (kDigits - 4);            // bits below the unit of the orders 0 to 3 (2^-38)
constexpr int kNotFinite = 1 << 20;                   // row exponent of a row that holds an infinity or NaN

// ------------------------------------------------------------------ split
// Eight CTAs per 64-row tile, a warp per row: the row's exponent from its largest
// magnitude, then eight values per lane into their digits (16-byte stores).
// Rows of up to 512 values are held in registers between the two steps, longer ones
// read again (from L1 / L2).  Bound: latency for the short rows, memory (8 bytes read,
// 16 written per value) for large operands.
__device__ __forceinline__ void split_load(const double* x, int k0, int k, bool vec, double (&v)[8]) {
  if (vec && k0 + 8 <= k) {
#pragma unroll
    for (int u = 0; u < 8; u += 2) *reinterpret_cast<double2*>(v + u) = *reinterpret_cast<const double2*>(x + k0 + u);
  } else {
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = k0 + u < k ? x[k0 + u] : 0.0;
  }
}
__device__ __forceinline__ unsigned exponent_field(double v) {
  return unsigned((__double_as_longlong(v) >> 52) & 0x7FF);
}
// eight values to digits; field: the row's largest exponent field (at least 1)
__device__ __forceinline__ void split_store(const double (&v)[8], int field, bool finite, uint8_t* dst, int k0) {
  uint32_t out[kDigits][4];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    long long F = 0;  // round(x 2^(kFracBits - e))
    if (finite) {
      const long long b = __double_as_longlong(v[u]);
      const int f = int((b >> 52) & 0x7FF);
      const long long m = (b & 0xFFFFFFFFFFFFFll) | (f ? 1ll << 52 : 0ll);
      const int sh = max(f, 1) - field + kFracBits - 53;
      if (sh >= 0) F = m << sh;
      else if (sh >= -54) F = (m + (1ll << (-sh - 1))) >> -sh;
      if (b < 0) F = -F;
    }
#pragma unroll
    for (int s = kDigits - 1; s >= 0; --s) {
      const int d = s > 0 ? int(int8_t(F & 0xFF)) : int(F);
      F = (F - d) >> 8;
      // d as a float by the spacing of floats near 1.5 2^23 (no conversion unit); exact in bf16
      const uint32_t h = __float_as_uint(__fsub_rn(__uint_as_float(0x4B400000u + unsigned(d)), 12582912.0f)) >> 16;
      if (u & 1) out[s][u >> 1] |= h << 16;
      else out[s][u >> 1] = h;
    }
  }
  uint8_t* q = dst + int64_t(k0 >> 5) * kChunkBytes + ((k0 >> 3) & 3) * 128;
#pragma unroll
  for (int s = 0; s < kDigits; ++s)
    *reinterpret_cast<uint4*>(q + s * kBlkBytes) = make_uint4(out[s][0], out[s][1], out[s][2], out[s][3]);
}

__global__ void __launch_bounds__(256) emu_split_kernel(const EmuSplit* __restrict__ tasks, const double* Ab,
                                                        const double* Bb, uint8_t* scratch) {
  const EmuSplit tk = tasks[blockIdx.x >> 3];
  const int lane = threadIdx.x & 31, r = int(blockIdx.x & 7) * 8 + int(threadIdx.x >> 5);
  chain_wait();
  if (r >= tk.rows) return;
  const double* x = (tk.buf ? Bb : Ab) + tk.src + int64_t(r) * tk.ld;
  const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  uint8_t* dst = scratch + tk.dst + (r >> 3) * 512 + (r & 7) * 16;
  double v[2][8];
  unsigned top = 0;  // largest exponent field
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    split_load(x, 8 * lane + 256 * h, tk.k, vec, v[h]);
#pragma unroll
    for (int u = 0; u < 8; ++u) top = max(top, exponent_field(v[h][u]));
  }
#pragma unroll 4
  for (int k = 512 + lane; k < tk.k; k += 32) top = max(top, exponent_field(x[k]));
  top = __reduce_max_sync(0xffffffffu, top);
  const bool finite = top != 0x7FF;
  const int field = max(int(top), 1);
  if (lane == 0) reinterpret_cast<int*>(scratch)[tk.exp + r] = finite ? field - 1022 : kNotFinite;
#pragma unroll
  for (int h = 0; h < 2; ++h)
    if (8 * lane + 256 * h < 32 * tk.nch) split_store(v[h], field, finite, dst, 8 * lane + 256 * h);
  for (int k0 = 512 + 8 * lane; k0 < 32 * tk.nch; k0 += 256) {
    split_load(x, k0, tk.k, vec, v[0]);
    split_store(v[0], field, finite, dst, k0);
  }
}

// ---------------------------------------------------------------- product
// shared-memory matrix descriptor: K-major, no swizzle; 8 x 16-byte core matrices
// 128 B apart along k, 8-row groups 512 B apart
__device__ __forceinline__ uint64_t emu_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= uint64_t((saddr & 0x3FFFFu) >> 4);
  d |= uint64_t(128 >> 4) << 16;
  d |= uint64_t(512 >> 4) << 32;
  d |= uint64_t(1) << 46;  // descriptor version
  return d;
}
// instruction descriptor: D F32, A/B BF16, both K-major, N = 64, M = 128
constexpr uint32_t kEmuIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((64u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void emu_mma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(kEmuIdesc), "r"(acc));
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(mbar)
               : "memory");
}

// (hi 2^kLoBits + lo) 2^e in FP64 for |hi| < 2^54, |lo| < 2^62: the leading 62 bits of the
// sum (all of them up to 2^62), converted with one rounding
__device__ __forceinline__ double emu_value(long long hi, long long lo, int e) {
  hi += lo >> kLoBits;
  const long long frac = lo & ((1ll << kLoBits) - 1);
  const int bits = 64 - __clzll(hi < 0 ? -hi : hi);                 // |hi| < 2^bits
  const int drop = bits > 62 - kLoBits ? bits - (62 - kLoBits) : 0;  // low bits of frac left out
  const long long v = hi * (1ll << (kLoBits - drop)) + (frac >> drop);
  e += drop;
  if (v == 0) return 0.0;
  const double d = double(v);
  const long long b = __double_as_longlong(d);
  const int f = int((b >> 52) & 0x7FF) + e;
  if (f > 0 && f < 0x7FF) return __longlong_as_double(b + (static_cast<long long>(e) << 52));
  return scalbn(d, e);
}

template <int MODE>
__global__ void __launch_bounds__(kEmuThreads, 1) emu_gemm_kernel(const EmuTask* __restrict__ tasks,
                                                                  const uint8_t* scratch, double* Cb, int* err,
                                                                  unsigned long long wait_ns) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full[kEmuStages], consumed[kEmuStages], dready, dfree, done;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag, mma_issued;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const EmuTask tk = tasks[blockIdx.x];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < kEmuStages; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[s])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&consumed[s])));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&dready)));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&done)));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&dfree)), "r"(kEpiWarps));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_flag = 0;
    mma_issued = 0;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    asm volatile("tcgen05.fence::before_thread_sync;");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_slot;
  chain_wait();
  const int nk = tk.k1 - tk.k0;                       // chunks
  const int nw = (nk + kWindow - 1) / kWindow;        // windows between drains

  auto wait = [&](uint64_t* bar, uint32_t parity, bool honor_abort, unsigned long long limit) -> bool {
    if (mbar_try(smem_u32(bar), parity)) return true;
    const unsigned long long t0 = now_ns();
    while (!mbar_try(smem_u32(bar), parity)) {
      if (honor_abort && *(volatile int*)&abort_flag) return false;
      if (now_ns() - t0 > limit) {
        atomicExch(&abort_flag, 1);
        return false;
      }
    }
    return true;
  };

  if (warp < kEpiWarps) {
    // ---------------- epilogue: lanes 32 (w % 4) .., output columns 16 (w / 4) ..
    const uint32_t lane_base = uint32_t((warp & 3) * 32) << 16;
    const int col0 = (warp >> 2) * 16;
    long long hi[16], lo[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) hi[c] = lo[c] = 0;
    bool ok = true;
    for (int w = 0; w < nw; ++w) {
      ok = __all_sync(0xffffffffu, wait(&dready, uint32_t(w & 1), true, wait_ns));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
      for (int o = 0; o < kDigits; ++o) {
        uint32_t r[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(tmem + lane_base + uint32_t(64 * o + col0)));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (o == kDigits - 1) {  // everything read: the next window may overwrite the accumulators
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&dfree));
        }
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          const int v = __float2int_rn(__uint_as_float(r[c]));
          if (o < 4) hi[c] += static_cast<long long>(v) * (1 << (24 - 8 * o));
          else lo[c] += static_cast<long long>(v) * (1 << (8 * (kDigits - 1 - o)));
        }
      }
    }
    chain_trigger();
    const int row = (warp & 3) * 32 + lane;
    if (ok && row < tk.m && col0 < tk.n) {
      const int* exps = reinterpret_cast<const int*>(scratch);
      const int ea = exps[tk.ea + row];
      double* dst = Cb + tk.c + int64_t(row) * tk.ldc + col0;
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        if (col0 + c >= tk.n) break;
        const int eb = exps[tk.eb + col0 + c];
        double v = emu_value(hi[c], lo[c], ea + eb - 38 - kLoBits);
        if (ea == kNotFinite || eb == kNotFinite) v = __longlong_as_double(0x7FF8000000000000ll);
        if (MODE == kSub) dst[c] -= v;
        else if (MODE == kStore) dst[c] = v;
        else if (MODE == kNegStore) dst[c] = -v;
        else dst[c] += v;
      }
    }
  } else if (warp == kEpiWarps) {
    // ---------------- loader: one thread issues the stage's bulk copies
    if (lane == 0) {
      int issued = 0;
      for (int t = 0; t < nk; ++t) {
        const int s = t % kEmuStages;
        if (t >= kEmuStages && !wait(&consumed[s], uint32_t(((t - kEmuStages) / kEmuStages) & 1), true, wait_ns)) break;
        const uint32_t d0 = smem_u32(smem + s * kStageBytes), fb = smem_u32(&full[s]);
        const uint8_t* a = scratch + tk.a + int64_t(tk.k0 + t) * kChunkBytes;
        mbar_expect_tx(fb, kStageBytes);
#pragma unroll
        for (int p = 0; p < kDigits; ++p) {
          bulk_load(d0 + p * 2 * kBlkBytes, a + p * kBlkBytes, kBlkBytes, fb);
          bulk_load(d0 + p * 2 * kBlkBytes + kBlkBytes, a + tk.a_step + p * kBlkBytes, kBlkBytes, fb);
        }
        bulk_load(d0 + kStageA, scratch + tk.b + int64_t(tk.k0 + t) * kChunkBytes, kChunkBytes, fb);
        issued = t + 1;
      }
      // copies still in flight (a failed wait ended the loop early) must land first
      for (int t = issued - kEmuStages > 0 ? issued - kEmuStages : 0; t < issued; ++t)
        wait(&full[t % kEmuStages], uint32_t((t / kEmuStages) & 1), false, kEmuWaitNs);
    }
  } else if (lane == 0) {
    // ---------------- MMA issuer
    for (int t = 0; t < nk; ++t) {
      const int s = t % kEmuStages, w = t / kWindow;
      if (t % kWindow == 0 && w > 0) {
        if (!wait(&dfree, uint32_t((w - 1) & 1), true, wait_ns)) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
      }
      if (!wait(&full[s], uint32_t((t / kEmuStages) & 1), true, wait_ns)) break;
      const uint32_t sa = smem_u32(smem + s * kStageBytes), sb = sa + kStageA;
#pragma unroll
      for (int ks = 0; ks < 2; ++ks)
#pragma unroll
        for (int o = 0; o < kDigits; ++o)
#pragma unroll
          for (int i = 0; i <= o; ++i)
            emu_mma(tmem + 64 * o, emu_desc(sa + i * 2 * kBlkBytes + ks * 256),
                    emu_desc(sb + (o - i) * kBlkBytes + ks * 256), (t % kWindow > 0 || ks > 0 || i > 0) ? 1u : 0u);
      mma_issued = 1;
      mma_commit(smem_u32(&consumed[s]));
      if (t % kWindow == kWindow - 1 || t == nk - 1) mma_commit(smem_u32(&dready));
    }
    if (mma_issued) mma_commit(smem_u32(&done));  // also after a failed wait: tells when every MMA is done
  }
  __syncthreads();
  if (tid == 0 && abort_flag) {
    atomicExch(err, 1);
    if (mma_issued) wait(&done, 0u, false, kEmuWaitNs);  // the MMAs read shared memory and write TMEM
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

template <int MODE>
void launch_emu(const EmuTask* t, int n, const uint8_t* scratch, double* C, int* err, cudaStream_t st,
                unsigned long long wait_ns) {
  allow_smem<emu_gemm_kernel<MODE>>(kEmuSmem);
  launch_chained(emu_gemm_kernel<MODE>, n, kEmuThreads, kEmuSmem, st, t, scratch, C, err, wait_ns);
}

}  // namespace

void launch_emu_gemm(const EmuSplit* splits, int nsplits, const EmuTask* tasks, int ntasks, const double* A,
                     const double* B, double* C, int mode, uint8_t* scratch, int* err, cudaStream_t st,
                     unsigned long long wait_ns) {
  if (ntasks <= 0) return;
  launch_chained(emu_split_kernel, 8 * nsplits, 256, 0, st, splits, A, B, scratch);
  switch (mode) {
    case kSub: launch_emu<kSub>(tasks, ntasks, scratch, C, err, st, wait_ns); break;
    case kStore: launch_emu<kStore>(tasks, ntasks, scratch, C, err, st, wait_ns); break;
    case kNegStore: launch_emu<kNegStore>(tasks, ntasks, scratch, C, err, st, wait_ns); break;
    default: launch_emu<kAdd>(tasks, ntasks, scratch, C, err, st, wait_ns); break;
  }
}

}  // namespace spde
