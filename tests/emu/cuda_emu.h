// The few CUDA device facilities that k_icp.cu uses, for a host compiler: one
// OS thread per CUDA thread, barriers as pthread barriers, warp exchanges
// through memory between two barriers of the warp's threads.  Shared memory is
// static storage, so a translation unit that includes a kernel is one block.
#pragma once
#include <math.h>
#include <pthread.h>
#include <sched.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <functional>
#include <string>
#include <thread>
#include <type_traits>
#include <vector>

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#undef __shared__
#define __shared__ static
#undef __global__
#define __global__
#undef __launch_bounds__
#define __launch_bounds__(...)
#undef __noinline__
#define __noinline__ __attribute__((noinline))

// called before an atomic operation on a counter (a test may hold a block there)
extern std::function<void(const void*)> emu_before_atomic;

namespace {

constexpr int kEmuThreads = 256;
thread_local uint3 threadIdx, blockIdx;

struct EmuBarrier {
  pthread_barrier_t b;
  explicit EmuBarrier(unsigned n) { pthread_barrier_init(&b, nullptr, n); }
  void wait() { pthread_barrier_wait(&b); }
};
struct EmuWarp {
  EmuBarrier bar{32};
  uint64_t v[32];
};
EmuBarrier emu_block(kEmuThreads), emu_named(64);
EmuWarp emu_warps[kEmuThreads / 32];

inline EmuWarp& emu_warp() { return emu_warps[threadIdx.x >> 5]; }
inline int emu_lane() { return (int)(threadIdx.x & 31); }
// every lane's value, to a function of the 32
template <class T, class F>
inline auto emu_exchange(T v, F&& f) {
  EmuWarp& w = emu_warp();
  uint64_t bits = 0;
  memcpy(&bits, &v, sizeof(T));
  w.v[emu_lane()] = bits;
  w.bar.wait();
  auto at = [&](int lane) {
    T r;
    memcpy(&r, &w.v[lane & 31], sizeof(T));
    return r;
  };
  const auto r = f(at);
  w.bar.wait();
  return r;
}

inline void __syncthreads() { emu_block.wait(); }
inline void emu_named_barrier() { emu_named.wait(); }
inline void __syncwarp() { emu_warp().bar.wait(); }
inline void __threadfence() { __atomic_thread_fence(__ATOMIC_SEQ_CST); }
inline void __nanosleep(unsigned) { sched_yield(); }

template <class T>
inline T __shfl_sync(unsigned, T v, int src) {
  return emu_exchange(v, [&](auto at) { return at(src); });
}
template <class T>
inline T __shfl_xor_sync(unsigned, T v, int m) {
  return emu_exchange(v, [&](auto at) { return at(emu_lane() ^ m); });
}
inline unsigned __ballot_sync(unsigned, bool p) {
  return emu_exchange(p, [&](auto at) {
    unsigned m = 0u;
    for (int k = 0; k < 32; k++) m |= at(k) ? 1u << k : 0u;
    return m;
  });
}
inline bool __all_sync(unsigned m, bool p) { return __ballot_sync(m, p) == 0xffffffffu; }
template <class T>
inline T __reduce_add_sync(unsigned, T v) {
  return emu_exchange(v, [&](auto at) {
    T s = 0;
    for (int k = 0; k < 32; k++) s += at(k);
    return s;
  });
}

template <class T>
inline T atomicAdd(T* p, T v) {
  if (emu_before_atomic) emu_before_atomic(p);
  return __atomic_fetch_add(p, v, __ATOMIC_SEQ_CST);
}
template <class T>
inline T atomicExch(T* p, T v) {
  return __atomic_exchange_n(p, v, __ATOMIC_SEQ_CST);
}
inline uint32_t atomicOr(uint32_t* p, uint32_t v) { return __atomic_fetch_or(p, v, __ATOMIC_SEQ_CST); }
template <class T>
inline T __ldg(const T* p) {
  return *p;
}
template <class T>
inline T __ldcg(const T* p) {
  return *p;
}
using std::max;
using std::min;
inline int __ffs(unsigned v) { return __builtin_ffs((int)v); }
inline uint32_t __float_as_uint(float f) {
  uint32_t u;
  memcpy(&u, &f, 4);
  return u;
}
inline float __uint_as_float(uint32_t u) {
  float f;
  memcpy(&f, &u, 4);
  return f;
}
inline uint64_t emu_bits(double d) {
  uint64_t u;
  memcpy(&u, &d, 8);
  return u;
}
inline int __double2hiint(double d) { return (int)(emu_bits(d) >> 32); }
inline int __double2loint(double d) { return (int)(uint32_t)emu_bits(d); }
inline double __hiloint2double(int hi, int lo) {
  const uint64_t u = (uint64_t)(uint32_t)hi << 32 | (uint32_t)lo;
  double d;
  memcpy(&d, &u, 8);
  return d;
}
inline long long __double_as_longlong(double d) { return (long long)emu_bits(d); }

// runs f as every thread of block b (threads: 32 or kEmuThreads)
template <class F>
inline void emu_run(int b, int threads, F f) {
  std::vector<std::thread> ts;
  for (int t = 0; t < threads; t++)
    ts.emplace_back([=] {
      threadIdx = make_uint3((unsigned)t, 0, 0);
      blockIdx = make_uint3((unsigned)b, 0, 0);
      f();
    });
  for (auto& t : ts) t.join();
}

}  // namespace
