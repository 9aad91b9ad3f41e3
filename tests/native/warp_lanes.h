// Test-only: a warp's 32 lanes on the host.  Each lane is a coroutine with a
// stack of its own; at a warp-wide operation it leaves its value and waits
// until all lanes have left theirs, so device code written for one warp runs
// as it is (compiled by g++, without divergence inside the operations).
// Several warps run side by side: __nanosleep gives the turn to another, and a
// schedule of the caller's says who is next.  Defines the CUDA names that
// csrc/align_warp.cuh uses; include it first.
#pragma once
#include <csetjmp>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <memory>
#include <type_traits>
#include <vector>
#include <ucontext.h>

namespace lanes {

constexpr size_t STACK = 256 << 10;

struct Warp {
  struct Lane {
    jmp_buf at;
    std::unique_ptr<char[]> stack;
    bool started = false, done = false, waits = false;
    unsigned ops = 0;  // warp-wide operations so far: their values alternate between two rows
  };
  Lane lane[32];
  uint64_t row[2][32];
  std::function<void()> body;
  bool done = false;
};

inline Warp *g_warp = nullptr;  // whose turn it is
inline int g_lane = 0;
inline jmp_buf g_turn;          // the scheduler
inline ucontext_t g_back;

inline std::function<void()> g_on_wake;  // called when a lane has slept

inline void leave() {
  Warp::Lane &l = g_warp->lane[g_lane];
  if (_setjmp(l.at) == 0) _longjmp(g_turn, 1);
}

inline void enter() {
  g_warp->body();
  g_warp->lane[g_lane].done = true;
  _longjmp(g_turn, 1);
}

// One turn of a warp: every lane up to its next operation, sleep or end.
inline void turn(Warp &w) {
  bool all = true, live = false;
  for (auto &l : w.lane) {
    all = all && (l.waits || l.done);
    live = live || !l.done;
  }
  if (!live) {
    w.done = true;
    return;
  }
  if (all)
    for (auto &l : w.lane) l.waits = false;
  for (int i = 0; i < 32; i++) {
    Warp::Lane &l = w.lane[i];
    if (l.done || l.waits) continue;
    g_warp = &w;
    g_lane = i;
    if (_setjmp(g_turn) == 0) {
      if (l.started) _longjmp(l.at, 1);
      l.started = true;
      l.stack.reset(new char[STACK]);
      static ucontext_t c;  // (static: it outlives the jump out of this frame)
      getcontext(&c);
      c.uc_stack.ss_sp = l.stack.get();
      c.uc_stack.ss_size = STACK;
      c.uc_link = nullptr;
      makecontext(&c, enter, 0);
      swapcontext(&g_back, &c);
    }
  }
}

// The values of all lanes, in lane order, once every lane is here.
template <class T>
const uint64_t *gather(T v) {
  static_assert(sizeof(T) <= 8, "a lane's value has at most 64 bits");
  Warp::Lane &l = g_warp->lane[g_lane];
  uint64_t *row = g_warp->row[l.ops++ & 1];
  row[g_lane] = 0;
  memcpy(&row[g_lane], &v, sizeof(T));
  l.waits = true;
  leave();
  return row;
}
template <class T>
T value(uint64_t bits) {
  T v;
  memcpy(&v, &bits, sizeof(T));
  return v;
}
template <class T, class F>
T fold(T v, F f) {
  const uint64_t *r = gather(v);
  T x = value<T>(r[0]);
  for (int i = 1; i < 32; i++) x = f(x, value<T>(r[i]));
  return x;
}
struct Id {
  int x;
};

}  // namespace lanes

#define __device__
#define __host__
#define __noinline__ __attribute__((noinline))
#define __forceinline__ inline
#define __align__(n) __attribute__((aligned(n)))
#define threadIdx (lanes::Id{lanes::g_lane})

// (the SM's id, which no test reads: the assembler skips the instruction)
__asm__(".macro mov.u32 a:vararg\n.endm\n");

struct __attribute__((aligned(16))) int4 {
  int x, y, z, w;
};
inline int4 make_int4(int x, int y, int z, int w) { return int4{x, y, z, w}; }

template <class T> T __shfl_sync(unsigned, T v, int src) { return lanes::value<T>(lanes::gather(v)[src & 31]); }
template <class T> T __shfl_up_sync(unsigned, T v, unsigned d) {
  const int l = lanes::g_lane;
  return lanes::value<T>(lanes::gather(v)[l >= (int)d ? l - (int)d : l]);
}
template <class T> T __shfl_xor_sync(unsigned, T v, int m) {
  const int l = lanes::g_lane;
  return lanes::value<T>(lanes::gather(v)[(l ^ m) & 31]);
}
inline unsigned __ballot_sync(unsigned, bool p) {
  const uint64_t *r = lanes::gather((int)p);
  unsigned m = 0;
  for (int i = 0; i < 32; i++) m |= (unsigned)(r[i] != 0) << i;
  return m;
}
inline bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0; }
inline bool __all_sync(unsigned m, bool p) { return __ballot_sync(m, p) == 0xffffffffu; }
template <class T> T __reduce_max_sync(unsigned, T v) { return lanes::fold(v, [](T a, T b) { return a > b ? a : b; }); }
template <class T> T __reduce_min_sync(unsigned, T v) { return lanes::fold(v, [](T a, T b) { return a < b ? a : b; }); }
inline int __reduce_add_sync(unsigned, int v) {
  return (int)lanes::fold((unsigned)v, [](unsigned a, unsigned b) { return a + b; });
}
inline unsigned __reduce_add_sync(unsigned, unsigned v) {
  return lanes::fold(v, [](unsigned a, unsigned b) { return a + b; });
}
inline unsigned __reduce_xor_sync(unsigned, unsigned v) {
  return lanes::fold(v, [](unsigned a, unsigned b) { return a ^ b; });
}
inline unsigned __reduce_or_sync(unsigned, unsigned v) {
  return lanes::fold(v, [](unsigned a, unsigned b) { return a | b; });
}
template <class T> unsigned __match_any_sync(unsigned, T v) {
  const uint64_t *r = lanes::gather(v);
  unsigned m = 0;
  for (int i = 0; i < 32; i++) m |= (unsigned)(r[i] == r[lanes::g_lane]) << i;
  return m;
}
inline void __syncwarp() { lanes::gather(0); }
inline void __threadfence() {}
inline void __nanosleep(unsigned) {
  lanes::leave();
  if (lanes::g_on_wake) lanes::g_on_wake();
}

inline int __popc(uint32_t v) { return __builtin_popcount(v); }
inline int __clz(int v) { return v ? __builtin_clz((unsigned)v) : 32; }
inline int __ffs(int v) { return __builtin_ffs(v); }
inline uint32_t __brev(uint32_t v) {
  uint32_t r = 0;
  for (int i = 0; i < 32; i++) r |= (v >> i & 1) << (31 - i);
  return r;
}
inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t s) {
  return (uint32_t)(((uint64_t)hi << 32 | lo) << (s & 31) >> 32);
}
inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s) {
  return (uint32_t)(((uint64_t)hi << 32 | lo) >> (s & 31));
}
template <class T> T __ldg(const T *p) { return *p; }
template <class T> T __ldcg(const T *p) { return *p; }
template <class T, class U> T atomicAdd(T *p, U v) {
  const T o = *p;
  *p = (T)(o + v);
  return o;
}
template <class T> T atomicCAS(T *p, T want, T v) {
  const T o = *p;
  if (o == want) *p = v;
  return o;
}
template <class T, class U> T atomicExch(T *p, U v) {
  const T o = *p;
  *p = (T)v;
  return o;
}
template <class A, class B> std::common_type_t<A, B> min(A a, B b) {
  using T = std::common_type_t<A, B>;
  return (T)a < (T)b ? (T)a : (T)b;
}
template <class A, class B> std::common_type_t<A, B> max(A a, B b) {
  using T = std::common_type_t<A, B>;
  return (T)a > (T)b ? (T)a : (T)b;
}
