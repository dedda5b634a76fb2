// Kernel launch interfaces shared by the CUDA translation units.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <atomic>
#include <cstdint>

namespace spde {

// One output tile of a batched product C (op)= A * B' over K.
// A is addressed as A[i*lda + k] (arow) or A[k*lda + i] (acol);
// B as B[j*ldb + k] (brow) or B[k*ldb + j] (bcol).  Offsets are in elements
// relative to the base pointers passed at launch.
struct GemmTask {
  int64_t a, b, c;
  int lda, ldb, ldc;
  int m, n, k;
  // cluster-pair tasks (256 x 256 tiles, tc_gemm.cu): tensor-map index of the
  // A / B operand (-1: loaded by cp.async) and the TMA coordinates (column,
  // row) of the task's first element in that map
  int amap = -1, bmap = -1;
  int ax = 0, ay = 0, bx = 0, by = 0;
  int pair = 0;
};

// Kernels of a schedule are launched as dependents of their predecessor in the
// stream: a kernel may be resident before the predecessor has finished (from the
// moment all its blocks have called chain_trigger or ended), reads only what the
// plan's set-up wrote until chain_wait, and every block calls chain_wait, so that a
// finished kernel implies finished predecessors.  Only what the set-up wrote is
// __restrict__: the predecessor still writes the rest while the kernel is resident, and the
// qualifier would let its loads move above chain_wait or through the read-only cache.  The trigger stands before a kernel's
// last stores: earlier, waiting blocks would hold SMs that another stream can use.
// Measured on evaluations (without / with): 16 x 16 x 8 2.00 / 1.74 ms, 47 x 39 x 13
// 7.36 / 6.62 ms, 100 x 100 x 24 74.8 / 73.1 ms; 256 draws at 100 x 100 x 24 34.3 / 32.0 ms.
#ifdef __CUDACC__
__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void chain_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#endif
template <typename... P, typename... A>
inline void launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Dynamic shared memory above 48 KB is granted per kernel and device: on its first launch on
// each (plans may live on several devices and launch from several threads)
template <auto Kernel>
inline void allow_smem(int bytes) {
  static std::atomic<uint64_t> granted{0};
  int dev = 0;
  cudaGetDevice(&dev);
  const uint64_t bit = dev < 64 ? uint64_t(1) << dev : 0;
  if (granted.load(std::memory_order_acquire) & bit) return;
  cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  granted.fetch_or(bit, std::memory_order_release);
}

// an integer constant as a type (selects a kernel's template argument in a lambda)
template <int N>
struct IntC {
  static constexpr int value = N;
};

enum GemmMode { kSub = 0, kStore = 1, kNegStore = 2, kAdd = 3 };
enum GemmLayout { kRow = 0, kCol = 1 };

// Diagonal-block task: factor the w x w block at `a` (row stride lda) in place,
// write its inverse to `dinv` (row stride nbk), record sum(log pivot).
struct DiagTask {
  int64_t a;
  int64_t dinv;
  int lda;
  int w;
  int front;
};

// Extend-add task: rows [r0, r1) of a front (positions, separator first).
struct ExtendTask {
  int front;
  int r0, r1;
};

struct DevFront {
  int64_t p_off, u_off, z_off, b_off, d_off;
  int64_t i_off;   // first entry of the front's positions in the extend-add source maps
  int64_t w_base;  // offset (per right-hand side) of this front's solve vectors in its depth pool
  int s0, ns, nb, ld, ldu, ldz, parent, depth;
  int child[2];
};

// product paths: CUDA-core tiles, tensor-core tiles (FP32 only), narrow (n <= 8
// columns), panel solve (FP32: m <= 128, n <= 64, k <= 64; CUDA-core tiles
// otherwise), 256 x 256 tiles on a cluster pair of tensor-core CTAs (FP32)
enum GemmPath { kPathSimt = 0, kPathTensor = 1, kPathNarrow = 2, kPathPanel = 3, kPathPair = 4 };
constexpr int kPairTile = 256;
// default wall-clock limit of every bounded wait in the tensor-core kernels
constexpr unsigned long long kTcWaitNs = 2000000000ull;
constexpr int kNarrowMaxN = 8;

// nmax bounds the tasks' n on the narrow path (1 selects the one-column kernel).
template <typename T>
void launch_gemm(const GemmTask* tasks, int ntasks, const T* A, const T* B, T* C, int mode, int alayout,
                 int blayout, cudaStream_t st, int path = kPathTensor, int nmax = kNarrowMaxN,
                 unsigned long long wait_ns = kTcWaitNs);

// tcgen05 path for FP32 (tc_gemm.cu); tc_gemm_take_error returns and clears the
// bounded-wait error flag of that kernel, read through `pinned` (page-locked host
// memory, so that the copy does not serialise with other host threads' copies).
void launch_gemm_tc(const GemmTask* tasks, int ntasks, const float* A, const float* B, float* C, int mode, int al,
                    int bl, cudaStream_t st, unsigned long long wait_ns = kTcWaitNs);
// cluster-pair path (row-major A and B): one 2-CTA cluster per 256 x 256 task
void launch_gemm_pair(const GemmTask* tasks, int ntasks, const CUtensorMap* maps, const float* A, const float* B,
                      float* C, int mode, cudaStream_t st, unsigned long long wait_ns = kTcWaitNs);
// FP64 products on the tensor cores (emu_gemm.cu).  Split task: 64 rows (the last
// tile of an operand fewer) of a row-major operand in buffer A (buf 0) or B (1),
// k values each, into nch = ceil(k / 32) chunks of digits at byte dst of the
// scratch and row exponents at its int exp.  Product task: one 128 x 64 tile over the
// chunks [k0, k1); a / b: byte offsets of the operand tiles' digits, a_step: bytes
// from A's first 64-row tile to its second, ea / eb: their row exponents.
constexpr int kEmuDigits = 8;
constexpr int64_t kEmuChunkBytes = kEmuDigits * 4096;  // 64 rows x 32 values, all digits
constexpr int64_t kEmuExpBytes = 64 * 4;               // row exponents of 64 rows
struct EmuSplit {
  int64_t src, dst, exp;
  int ld, rows, k, nch, buf;
};
struct EmuTask {
  int64_t a, b, c, a_step, ea, eb;
  int ldc, m, n, k0, k1;
};
void launch_emu_gemm(const EmuSplit* splits, int nsplits, const EmuTask* tasks, int ntasks, const double* A,
                     const double* B, double* C, int mode, uint8_t* scratch, int* err, cudaStream_t st,
                     unsigned long long wait_ns = kTcWaitNs);
int tc_gemm_take_error(cudaStream_t st, int* pinned);
bool tc_gemm_enabled();

template <typename T>
void launch_potrf(const DiagTask* tasks, int ntasks, T* L, T* dinv, double* logpiv, int* err, cudaStream_t st);

template <typename T>
void launch_extend(const ExtendTask* tasks, int ntasks, const DevFront* fronts, const int* src0, const int* src1,
                   const T* U_child, T* L, T* U_parent, cudaStream_t st);

}  // namespace spde
