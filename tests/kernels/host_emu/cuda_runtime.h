// Stands in for the CUDA runtime header when a kernel's source is compiled for the host: one
// block runs as fibers on one host thread, each until it waits at a block or warp barrier, in
// an order the test chooses (emu::late_warp runs only when no other warp can).  Block barriers
// check that every thread waits at the same source line.  What a test does not run is declared
// only.
#pragma once
#include <math.h>
#include <stddef.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <ucontext.h>

#include <functional>
#include <type_traits>
#include <vector>

#define __device__
#define __host__
#define __global__
#define __shared__ static
#define __forceinline__ inline
#define __noinline__
#define __restrict__
#define __launch_bounds__(...)
#define __align__(n) __attribute__((aligned(n)))

struct dim3 {
  unsigned x = 1, y = 1, z = 1;
};
inline dim3 threadIdx, blockIdx, blockDim, gridDim;

namespace emu {
constexpr int kStack = 256 * 1024;
struct Fiber {
  ucontext_t ctx;
  std::vector<char> stack;
  bool finished = false;
  int block_line = 0;  // the source line of the block barrier it waits at, 0: none
  bool in_warp = false;
  int pred = 0;  // the value it brought to its warp's or the block's vote
  double carried[2];  // the values it brought to its warp's last two shuffles
  int shuffles = 0;
};
inline std::vector<Fiber> fibers;
inline ucontext_t scheduler;
inline int current = -1;
inline int late_warp = -1;
inline bool failed = false;
inline int block_or = 0;
inline std::vector<unsigned> warp_mask;
inline std::function<void()> body;
inline const char* shared_base = nullptr;

inline void entry() {
  body();
  fibers[current].finished = true;
  swapcontext(&fibers[current].ctx, &scheduler);
}
inline void yield() { swapcontext(&fibers[current].ctx, &scheduler); }

inline int block_sync(int line, int pred) {
  fibers[current].block_line = line;
  fibers[current].pred = pred;
  yield();
  return block_or;
}
inline unsigned warp_vote(int pred) {
  fibers[current].in_warp = true;
  fibers[current].pred = pred;
  yield();
  return warp_mask[current / 32];
}

inline double shuffle_xor(double v, int lanes) {
  Fiber& f = fibers[current];
  const int slot = f.shuffles++ & 1, partner = current ^ lanes;
  f.carried[slot] = v;
  warp_vote(0);
  return fibers[partner].carried[slot];
}

// Runs fn on `threads` threads of block `block`; false when barriers diverge or cannot complete.
inline bool run_block(int threads, int block, int grid, std::function<void()> fn) {
  body = std::move(fn);
  failed = false;
  blockDim.x = (unsigned)threads;
  gridDim.x = (unsigned)grid;
  blockIdx.x = (unsigned)block;
  fibers.assign((size_t)threads, Fiber{});
  warp_mask.assign((size_t)(threads / 32), 0u);
  for (auto& f : fibers) {
    f.stack.resize(kStack);
    getcontext(&f.ctx);
    f.ctx.uc_stack.ss_sp = f.stack.data();
    f.ctx.uc_stack.ss_size = f.stack.size();
    f.ctx.uc_link = nullptr;
    makecontext(&f.ctx, entry, 0);
  }
  auto runnable = [&](int t) {
    return !fibers[t].finished && fibers[t].block_line == 0 && !fibers[t].in_warp;
  };
  for (;;) {
    bool ran = false;
    for (int pass = 0; pass < 2 && !ran; pass++)
      for (int t = 0; t < threads; t++) {
        if ((t / 32 == late_warp) != (pass == 1) || !runnable(t)) continue;
        current = t;
        threadIdx.x = (unsigned)t;
        swapcontext(&scheduler, &fibers[t].ctx);
        ran = true;
      }
    // warp votes that every lane of a warp has reached
    for (int w = 0; w < threads / 32; w++) {
      unsigned m = 0;
      int in = 0;
      for (int l = 0; l < 32; l++) {
        const Fiber& f = fibers[w * 32 + l];
        in += f.in_warp;
        if (f.in_warp && f.pred) m |= 1u << l;
      }
      if (in < 32) continue;
      warp_mask[w] = m;
      for (int l = 0; l < 32; l++) fibers[w * 32 + l].in_warp = false;
      ran = true;
    }
    if (ran) continue;
    int waiting = 0, done = 0, line = 0, any = 0;
    bool same = true;
    for (auto& f : fibers) {
      done += f.finished;
      if (!f.block_line) continue;
      waiting++;
      any |= f.pred;
      if (line && f.block_line != line) same = false;
      line = f.block_line;
    }
    if (done == threads) return true;
    if (waiting + done < threads || done > 0 || !same) {
      fprintf(stderr, "block barrier: %d of %d threads wait, %d have returned%s\n", waiting, threads,
              done, same ? "" : ", at different barriers");
      failed = true;
      return false;
    }
    block_or = any;
    for (auto& f : fibers) f.block_line = 0;
  }
}
}  // namespace emu

#define __syncthreads() ((void)emu::block_sync(__LINE__, 0))
#define __syncthreads_or(p) emu::block_sync(__LINE__, (p) ? 1 : 0)
inline void __syncwarp(unsigned = 0xffffffffu) { emu::warp_vote(0); }
inline unsigned __ballot_sync(unsigned, int p) { return emu::warp_vote(p); }
inline int __any_sync(unsigned, int p) { return emu::warp_vote(p) != 0; }
inline int __all_sync(unsigned, int p) { return emu::warp_vote(p) == 0xffffffffu; }
inline double __shfl_xor_sync(unsigned, double v, int lanes) { return emu::shuffle_xor(v, lanes); }
inline int __ffs(unsigned m) { return __builtin_ffs((int)m); }
inline int __popc(unsigned m) { return __builtin_popcount(m); }
template <typename T>
T __ldcg(const T* p) {
  return *p;
}
template <typename T>
T __ldg(const T* p) {
  return *p;
}
inline double __longlong_as_double(long long v) {
  double d;
  memcpy(&d, &v, 8);
  return d;
}
inline long long __double_as_longlong(double d) {
  long long v;
  memcpy(&v, &d, 8);
  return v;
}
inline size_t __cvta_generic_to_shared(const void* p) { return (size_t)((const char*)p - emu::shared_base); }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __ddiv_rn(double a, double b) { return a / b; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fdiv_rn(float a, float b) { return a / b; }
inline void __threadfence() {}
// named by sources whose use of them no test runs
unsigned long long __shfl_xor_sync(unsigned, unsigned long long, int);
unsigned int __shfl_xor_sync(unsigned, unsigned int, int);
double __fma_rn(double, double, double);
float __fmaf_rn(float, float, float);
double __dmul_ru(double, double), __dmul_rd(double, double);
float __fmul_ru(float, float), __fmul_rd(float, float);
float __int_as_float(int);
int __float_as_int(float);
template <typename T>
T atomicAdd(T* p, T v) {
  const T old = *p;
  *p = old + v;
  return old;
}
template <typename T>
T atomicExch(T* p, T v) {
  const T old = *p;
  *p = v;
  return old;
}
