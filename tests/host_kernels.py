"""Runs CUDA kernels of this repository on the CPU, a block at a time, every thread a
coroutine that runs until its next barrier or shuffle.  Which thread goes next is the
caller's choice (`order`), so that what a kernel leaves to chance can be made to happen:
with "up" warp 0 runs as far as its barriers let it before warp 1 begins, with "down"
the last warp does.  Kernels with inline assembly in what they execute are not for this.
"""
import ctypes
import hashlib
import os
import re
import subprocess
import tempfile

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "spdepy_gb300", "csrc")

FLAGS = ["-std=c++17", "-O1", "-ffp-contract=off", "-fwrapv", "-w", "-shared", "-fPIC"]  # integers wrap as on the GPU

RUNTIME = r"""
#include <math.h>
#include <stdint.h>
#include <string.h>
#include <ucontext.h>
#include <algorithm>
#include <vector>
#define __device__
#define __global__
#define __host__
#define __restrict__
#define __forceinline__ inline
#define __align__(n) __attribute__((aligned(n)))
#define __launch_bounds__(...)
using std::max;
using std::min;
struct dim3h { int x, y, z; };
struct float2 { float x, y; };
struct alignas(16) float4 { float x, y, z, w; };
struct alignas(16) double2 { double x, y; };
inline float2 make_float2(float a, float b) { return {a, b}; }
inline float4 make_float4(float a, float b, float c, float d) { return {a, b, c, d}; }
namespace host {
struct Thread {
  ucontext_t ctx;
  std::vector<char> stack;
  dim3h tid;
  int state = 0;  // 0 runnable, 1 at the block's barrier, 2 at its warp's, 3 done
};
struct Block {
  std::vector<Thread> t;
  ucontext_t main;
  int cur = 0;
  dim3h bid, bdim, gdim;
  uint64_t slot[64][2][32];  // shuffles: per warp, by parity
  int parity[64 * 32];
  void (*body)(void*);
  void* arg;
};
extern Block* blk;
inline void yield(int state) {
  Thread& me = blk->t[blk->cur];
  me.state = state;
  swapcontext(&me.ctx, &blk->main);
}
inline void entry() {
  blk->body(blk->arg);
  yield(3);
}
inline void run(dim3h bid, dim3h gdim, int threads, bool up, void (*body)(void*), void* arg) {
  Block b;
  b.t.resize(threads);
  b.bid = bid; b.gdim = gdim; b.bdim = {threads, 1, 1};
  b.body = body; b.arg = arg;
  memset(b.parity, 0, sizeof(b.parity));
  blk = &b;
  for (int i = 0; i < threads; ++i) {
    Thread& t = b.t[i];
    t.stack.resize(1 << 17);
    t.tid = {i, 0, 0};
    getcontext(&t.ctx);
    t.ctx.uc_stack.ss_sp = t.stack.data();
    t.ctx.uc_stack.ss_size = t.stack.size();
    t.ctx.uc_link = &b.main;
    makecontext(&t.ctx, (void (*)())entry, 0);
  }
  const int warps = threads / 32;
  for (;;) {
    bool ran = false;
    for (int q = 0; q < warps && !ran; ++q) {
      const int w = up ? q : warps - 1 - q;
      int waiting = 0, done = 0;
      for (int l = 0; l < 32; ++l) {
        Thread& t = b.t[32 * w + l];
        if (t.state == 0) {
          b.cur = 32 * w + l;
          swapcontext(&b.main, &t.ctx);
          ran = true;
        }
        waiting += t.state == 2;
        done += t.state == 3;
      }
      if (waiting && waiting + done == 32) {
        for (int l = 0; l < 32; ++l)
          if (b.t[32 * w + l].state == 2) b.t[32 * w + l].state = 0;
        ran = true;
      }
    }
    if (ran) continue;
    int left = 0, at = 0;
    for (auto& t : b.t) { left += t.state != 3; at += t.state == 1; }
    if (!left) return;
    if (at != left) abort();  // part of the block waits where the others never come
    for (auto& t : b.t)
      if (t.state == 1) t.state = 0;
  }
}
}  // namespace host
#define threadIdx (host::blk->t[host::blk->cur].tid)
#define blockIdx (host::blk->bid)
#define blockDim (host::blk->bdim)
#define gridDim (host::blk->gdim)
inline void __syncthreads() { host::yield(1); }
inline void __syncwarp() { host::yield(2); }
inline void chain_wait() {}
inline void chain_trigger() {}
template <typename T>
inline T host_shfl(T v, int src) {
  host::Block* b = host::blk;
  const int me = b->cur, w = me >> 5, p = b->parity[me];
  b->parity[me] ^= 1;
  memcpy(&b->slot[w][p][me & 31], &v, sizeof(T));
  host::yield(2);
  T r;
  memcpy(&r, &b->slot[w][p][src], sizeof(T));
  return r;
}
template <typename T>
inline T __shfl_sync(unsigned, T v, int lane) { return host_shfl(v, lane); }
template <typename T>
inline T __shfl_xor_sync(unsigned, T v, int m) { return host_shfl(v, (host::blk->cur & 31) ^ m); }
template <typename T>
inline T __shfl_down_sync(unsigned, T v, int d) {
  const int l = host::blk->cur & 31;
  return host_shfl(v, l + d < 32 ? l + d : l);
}
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fdividef(float a, float b) { return a / b; }
inline float __fdiv_rn(float a, float b) { return a / b; }
inline float rsqrtf(float a) { return 1.0f / sqrtf(a); }
inline double rsqrt(double a) { return 1.0 / sqrt(a); }
inline int64_t __double_as_longlong(double v) { int64_t r; memcpy(&r, &v, 8); return r; }
inline double __longlong_as_double(int64_t v) { double r; memcpy(&r, &v, 8); return r; }
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int atomicCAS(int* p, int c, int v) { const int o = *p; if (o == c) *p = v; return o; }
inline unsigned atomicOr(uint32_t* p, uint32_t v) { const uint32_t o = *p; *p |= v; return o; }
"""


def section(source, begin, end):
    """The text of csrc/`source` from the line that starts with `begin` to the one before `end`."""
    with open(os.path.join(CSRC, source)) as f:
        text = f.read()
    i = text.index("\n" + begin) + 1
    return text[i:text.index("\n" + end, i) + 1]


def compile_host(parts, tail):
    """A library from sections of kernels (`parts`) and `tail`, host code that runs them."""
    code = "\n".join(parts)
    code = re.sub(r"asm( volatile)?\(.*?\);", ";", code, flags=re.S)
    code = code.replace("extern __shared__", "extern").replace("__shared__", "static")
    text = RUNTIME + "namespace host { Block* blk; }\n" + code + tail
    out = os.path.join(tempfile.gettempdir(), "host_kernels_%s.so" % hashlib.sha1((text + repr(FLAGS)).encode()).hexdigest()[:16])
    if not os.path.exists(out):
        with tempfile.TemporaryDirectory() as d:
            src, lib = os.path.join(d, "k.cpp"), os.path.join(d, "k.so")
            with open(src, "w") as f:
                f.write(text)
            subprocess.run(["g++", *FLAGS, src, "-o", lib], check=True)
            os.replace(lib, out)
    return ctypes.CDLL(out)
