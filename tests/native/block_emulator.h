// A CUDA block on one host thread, for tests of a kernel's barriers: every device thread is a fiber that runs until it
// waits (a block barrier or a warp's collective), and of the threads that can run the scheduler always takes the first
// in a given order of the warps and lanes. So a warp can be let run ahead of the others as far as its barriers allow, a
// schedule the device may pick too; code whose results depend on the order lacks a barrier. Asynchronous copies land
// when they are issued or, with `late`, when their thread waits for them: the earliest and the latest they may.
#pragma once
#include <cuda_runtime.h>
#include <ucontext.h>
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <functional>
#include <memory>
#include <vector>
#include <cstdio>

namespace emu {

constexpr size_t STACK = 256 * 1024;
struct Thread {
  ucontext_t ctx;
  std::unique_ptr<char[]> stack;
  int id = 0;
  enum { READY, BARRIER, WARP, ENDED } state = READY;
  unsigned generation = 0;  // warp collectives this thread has entered
  struct Copy { void* to; const void* from; size_t bytes; };
  std::vector<Copy> copies;  // not yet landed
};
struct Warp {
  uint64_t values[2][32];
  int arrived = 0;
};
struct Block {
  std::vector<Thread> threads;
  std::vector<Warp> warps;
  std::vector<int> order;  // the threads by priority
  ucontext_t home;
  Thread* self = nullptr;
  std::function<void()> body;
  bool late = false, deadlock = false;
};
inline Block*& block() { static Block* b = nullptr; return b; }

__attribute__((noinline)) inline void yield() {
  Block& b = *block();
  Thread* t = b.self;
  swapcontext(&t->ctx, &b.home);
  asm volatile("" ::: "memory");
}
inline void entry() {
  block()->body();
  block()->self->state = Thread::ENDED;
  yield();
}
// Every lane's value, once all 32 lanes of the warp are here.
inline const uint64_t* collect(uint64_t v) {
  Block& b = *block();
  Thread* t = b.self;
  Warp& w = b.warps[t->id / 32];
  const int side = t->generation++ & 1;
  w.values[side][t->id % 32] = v;
  if (++w.arrived == 32) {
    w.arrived = 0;
    for (int l = 0; l < 32; l++) { Thread& o = b.threads[t->id / 32 * 32 + l]; if (o.state == Thread::WARP) o.state = Thread::READY; }
  } else {
    t->state = Thread::WARP;
    yield();
  }
  return w.values[side];
}
inline void copy(void* to, const void* from, size_t bytes) {
  if (block()->late) block()->self->copies.push_back({to, from, bytes});
  else std::memcpy(to, from, bytes);
}
inline void land() {
  for (const Thread::Copy& c : block()->self->copies) std::memcpy(c.to, c.from, c.bytes);
  block()->self->copies.clear();
}
inline void barrier() { block()->self->state = Thread::BARRIER; yield(); }

// Runs `body` as `threads` device threads (whole warps). order 0: warps and lanes ascending; 1: both descending; k >= 2:
// warp k - 2 first, then ascending. False where the threads wait for one another forever.
inline bool run(int threads, int order, const std::function<void()>& body, bool late = false) {
  Block b;
  b.late = late;
  b.threads.resize(threads); b.warps.resize(threads / 32); b.body = body;
  block() = &b;
  for (int t = 0; t < threads; t++) {
    Thread& f = b.threads[t];
    f.id = t; f.stack.reset(new char[STACK]);
    getcontext(&f.ctx);
    f.ctx.uc_stack.ss_sp = f.stack.get(); f.ctx.uc_stack.ss_size = STACK; f.ctx.uc_link = &b.home;
    makecontext(&f.ctx, entry, 0);
    b.order.push_back(t);
  }
  if (order == 1) std::reverse(b.order.begin(), b.order.end());
  if (order >= 2) {
    const int w = (order - 2) % (threads / 32);
    std::stable_partition(b.order.begin(), b.order.end(), [w](int t) { return t / 32 == w; });
  }
  for (;;) {
    Thread* next = nullptr;
    for (int t : b.order) if (b.threads[t].state == Thread::READY) { next = &b.threads[t]; break; }
    if (next) { b.self = next; swapcontext(&b.home, &next->ctx); continue; }
    bool ended = true, all = true;
    for (const Thread& f : b.threads) { ended = ended && f.state == Thread::ENDED; all = all && (f.state == Thread::BARRIER || f.state == Thread::ENDED); }
    if (ended || !all) { b.deadlock = !ended; if(!ended) for (const Thread& f : b.threads) fprintf(stderr,"%d:%d(%u) ", f.id, (int)f.state, f.generation); break; }
    for (Thread& f : b.threads) if (f.state == Thread::BARRIER) f.state = Thread::READY;
  }
  block() = nullptr;
  return !b.deadlock;
}

template <class T> uint64_t bits(T v) { uint64_t u = 0; std::memcpy(&u, &v, sizeof(T)); return u; }
template <class T> T from(uint64_t u) { T v; std::memcpy(&v, &u, sizeof(T)); return v; }
struct Index { int x; };
struct Dim { unsigned x; };
inline Index thread_index() { return Index{block()->self->id}; }
inline Dim block_dim() { return Dim{(unsigned)block()->threads.size()}; }

}  // namespace emu

#define threadIdx (emu::thread_index())
#define blockDim (emu::block_dim())
#define __shared__ static
#define __global__ static
#define __device__
#define __constant__
#define __restrict__
#define __launch_bounds__(...)
#define __forceinline__ inline

inline int min(int a, int b) { return a < b ? a : b; }
inline int max(int a, int b) { return a > b ? a : b; }
inline void __syncthreads() { emu::barrier(); }
inline void __syncwarp() { emu::collect(0); }
template <class T> T __shfl_sync(unsigned, T v, int lane) { return emu::from<T>(emu::collect(emu::bits(v))[lane & 31]); }
template <class T> T __shfl_up_sync(unsigned, T v, int o) {
  const int lane = threadIdx.x & 31;
  return emu::from<T>(emu::collect(emu::bits(v))[lane >= o ? lane - o : lane]);
}
template <class T> T __shfl_xor_sync(unsigned, T v, int o) { return emu::from<T>(emu::collect(emu::bits(v))[(threadIdx.x & 31) ^ o]); }
inline unsigned __ballot_sync(unsigned, bool p) {
  const uint64_t* v = emu::collect(p);
  unsigned m = 0;
  for (int l = 0; l < 32; l++) m |= (unsigned)(v[l] != 0) << l;
  return m;
}
inline int __ffs(unsigned v) { return __builtin_ffs((int)v); }
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __clz(unsigned v) { return v ? __builtin_clz(v) : 32; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __dadd_rn(double a, double b) { return a + b; }
inline long long __double_as_longlong(double v) { return emu::from<long long>(emu::bits(v)); }
inline float __int_as_float(int v) { return emu::from<float>((uint32_t)v); }
inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
inline float __fdividef(float a, float b) { return a / b; }
inline float2 __fmul2_rn(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
inline float2 __fadd2_rn(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
inline float2 __ffma2_rn(float2 a, float2 b, float2 c) { return make_float2(std::fma(a.x, b.x, c.x), std::fma(a.y, b.y, c.y)); }
inline void cp_async4(float* to, const float* from) { emu::copy(to, from, 4); }
inline void cp_async16(void* to, const void* from) { emu::copy(to, from, 16); }
inline void cp_async_wait_all() { emu::land(); }
