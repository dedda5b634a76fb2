// Asynchronous copies, shared-memory barriers and tensor-core helpers.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "kernels.cuh"

namespace spde {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
               : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t mbar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(mbar), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// ------------------------------------------------- C tiles of the FP32 products
template <int MODE>
__device__ __forceinline__ float apply_mode(float old, float v) {
  if (MODE == kSub) return old - v;
  if (MODE == kStore) return v;
  if (MODE == kNegStore) return -v;
  return old + v;
}
// The C tile of an updating product into L2 while the mainloop runs
template <int COLS, int NT>
__device__ __forceinline__ void prefetch_c(const float* C, int64_t ldc, int m, int n, int ltid) {
  constexpr int kLines = COLS / 32;
  for (int e = ltid; e < m * kLines; e += NT) {
    const int r = e / kLines, c = 32 * (e - r * kLines);
    if (c < n) asm volatile("prefetch.global.L2 [%0];" ::"l"(C + r * ldc + c));
  }
}
// Rows warp, warp + NW, ... of an m x n tile (rows of `ld` floats in shared memory,
// COLS of them computed) into C, four rows in flight
template <int MODE, int COLS, int NW>
__device__ __forceinline__ void rows_to_global(const float* sm, int ld, float* C, int64_t ldc, int m, int n, int warp,
                                               int lane) {
  constexpr bool kRead = MODE == kSub || MODE == kAdd;
  const bool vec = ((reinterpret_cast<uintptr_t>(C) & 15) == 0) && (ldc & 3) == 0;
#pragma unroll 1
  for (int r0 = warp; r0 < m; r0 += 4 * NW) {
#pragma unroll
    for (int c0 = 0; c0 < COLS; c0 += 128) {
      const int c = c0 + 4 * lane;
      if (vec && c0 + 128 <= n) {
        float4 old[4];
        if (kRead) {
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (r0 + u * NW < m) old[u] = *reinterpret_cast<const float4*>(C + (r0 + u * NW) * ldc + c);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (r0 + u * NW < m) {
            const float4 v = *reinterpret_cast<const float4*>(sm + (r0 + u * NW) * ld + c);
            *reinterpret_cast<float4*>(C + (r0 + u * NW) * ldc + c) =
                make_float4(apply_mode<MODE>(old[u].x, v.x), apply_mode<MODE>(old[u].y, v.y),
                            apply_mode<MODE>(old[u].z, v.z), apply_mode<MODE>(old[u].w, v.w));
          }
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {  // one column per lane
          const int cj = c0 + lane + 32 * j;
          float old[4];
          if (kRead) {
#pragma unroll
            for (int u = 0; u < 4; ++u)
              if (r0 + u * NW < m && cj < n) old[u] = C[(r0 + u * NW) * ldc + cj];
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (r0 + u * NW < m && cj < n)
              C[(r0 + u * NW) * ldc + cj] = apply_mode<MODE>(old[u], sm[(r0 + u * NW) * ld + cj]);
        }
      }
    }
  }
}

}  // namespace spde
