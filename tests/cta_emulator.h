// Runs a CUDA kernel's CTA on the host, one fiber per thread, so that CPU tests can run the kernels of
// planning.cuh as they are and under any order of the warps: a warp runs until all its lanes wait at
// a CTA barrier (or have returned), then the next warp of the chosen order does. On a GPU any such
// interleaving can happen; code that needs another one lacks a barrier.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <ucontext.h>
#include <functional>
#include <vector>

namespace emu {

enum State { kRun, kWarp, kCta, kDone };

struct Fiber {
  ucontext_t at;
  std::vector<char> stack;
  State state = kRun;
};

struct Cta {
  std::vector<Fiber> fibers;
  std::vector<uint64_t> value;  // operand of a lane's warp step
  int current = 0;
  ucontext_t scheduler;
  std::function<void()> body;
  dim3 block, grid;
  uint3 block_id;
  int or_now = 0, or_last = 0;
};

inline Cta*& cta() {
  static Cta* c = nullptr;
  return c;
}

inline uint3 thread_id() { return {(unsigned)cta()->current, 0, 0}; }

inline void wait(State s) {
  Cta* c = cta();
  Fiber& f = c->fibers[c->current];
  f.state = s;
  swapcontext(&f.at, &c->scheduler);
}

inline void entry() {
  cta()->body();
  wait(kDone);
}

// Runs the lanes of one warp until every one waits at the CTA barrier or has returned.
inline void run_warp(Cta* c, int w) {
  const int a = 32 * w, b = a + 32 < (int)c->fibers.size() ? a + 32 : (int)c->fibers.size();
  for (;;) {
    for (int t = a; t < b; ++t) {
      if (c->fibers[t].state != kRun) continue;
      c->current = t;
      swapcontext(&c->scheduler, &c->fibers[t].at);
    }
    int at_step = 0;
    for (int t = a; t < b; ++t) at_step += c->fibers[t].state == kWarp;
    if (!at_step) return;
    if (at_step != b - a) {
      fprintf(stderr, "warp step without all lanes\n");
      abort();
    }
    for (int t = a; t < b; ++t) c->fibers[t].state = kRun;
  }
}

// One CTA of `threads` threads; `order` is a permutation of its warps.
inline void run_cta(int threads, dim3 grid, unsigned block, const std::vector<int>& order,
                    const std::function<void()>& body) {
  Cta c;
  c.fibers.resize(threads);
  c.value.resize(threads);
  c.body = body;
  c.block = dim3(threads);
  c.grid = grid;
  c.block_id = {block, 0, 0};
  cta() = &c;
  for (Fiber& f : c.fibers) {
    f.stack.resize(32 << 10);
    getcontext(&f.at);
    f.at.uc_stack.ss_sp = f.stack.data();
    f.at.uc_stack.ss_size = f.stack.size();
    makecontext(&f.at, entry, 0);
  }
  for (;;) {
    for (int w : order) run_warp(&c, w);
    int done = 0, waiting = 0;
    for (Fiber& f : c.fibers) (f.state == kDone ? done : waiting)++;
    if (!waiting) break;
    c.or_last = c.or_now;
    c.or_now = 0;
    for (Fiber& f : c.fibers)
      if (f.state == kCta) f.state = kRun;
  }
  cta() = nullptr;
}

// Puts v beside the other lanes' operands; two waits, so that a lane that runs ahead does not
// overwrite its operand before the others have read it.
template <typename T>
T exchange(T v, const std::function<T(const T*, int)>& read) {
  static_assert(sizeof(T) <= 8, "");
  Cta* c = cta();
  const int me = c->current, base = me / 32 * 32;
  c->value[me] = 0;
  __builtin_memcpy(&c->value[me], &v, sizeof(T));
  wait(kWarp);
  T lanes[32];
  for (int l = 0; l < 32; ++l) __builtin_memcpy(&lanes[l], &c->value[base + l], sizeof(T));
  const T r = read(lanes, me - base);
  wait(kWarp);
  return r;
}

}  // namespace emu

#undef __shared__
#undef __device__
#undef __host__
#undef __global__
#undef __forceinline__
#undef __launch_bounds__
#define __shared__ static  // (CTAs run one after the other)
#define __device__
#define __host__
#define __global__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define threadIdx (emu::thread_id())
#define blockIdx (emu::cta()->block_id)
#define blockDim (emu::cta()->block)
#define gridDim (emu::cta()->grid)

inline void __syncthreads() { emu::wait(emu::kCta); }
inline int __syncthreads_or(int p) {
  emu::cta()->or_now |= p != 0;
  emu::wait(emu::kCta);
  return emu::cta()->or_last;
}
template <typename T>
T __shfl_sync(unsigned, T v, int src) {
  return emu::exchange<T>(v, [=](const T* l, int) { return l[src & 31]; });
}
template <typename T>
T __shfl_up_sync(unsigned, T v, int o) {
  return emu::exchange<T>(v, [=](const T* l, int me) { return me >= o ? l[me - o] : l[me]; });
}
template <typename T>
T __shfl_xor_sync(unsigned, T v, int o) {
  return emu::exchange<T>(v, [=](const T* l, int me) { return l[me ^ o]; });
}
inline unsigned __ballot_sync(unsigned, int p) {
  return emu::exchange<unsigned>(p ? 1u : 0u, [](const unsigned* l, int) {
    unsigned m = 0;
    for (int i = 0; i < 32; ++i) m |= l[i] << i;
    return m;
  });
}
inline unsigned __reduce_max_sync(unsigned, unsigned v) {
  return emu::exchange<unsigned>(v, [](const unsigned* l, int) {
    unsigned m = 0;
    for (int i = 0; i < 32; ++i) m = l[i] > m ? l[i] : m;
    return m;
  });
}
template <typename T, typename U>
T atomicAdd(T* p, U v) {
  const T old = *p;
  *p = old + (T)v;
  return old;
}
template <typename T, typename U>
T atomicMax(T* p, U v) {
  const T old = *p;
  if ((T)v > old) *p = (T)v;
  return old;
}
inline int __clz(int v) { return v ? __builtin_clz((unsigned)v) : 32; }
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __ffs(int v) { return __builtin_ffs(v); }
inline void cudaTriggerProgrammaticLaunchCompletion() {}
inline void cudaGridDependencySynchronize() {}
template <typename T>
T min(T a, T b) { return b < a ? b : a; }
template <typename T>
T max(T a, T b) { return a < b ? b : a; }
