// Stand-ins that run device code of this library on host threads, so that the
// ordering of its accesses to shared variables can be checked on the CPU
// (ThreadSanitizer): one host thread per CUDA thread, a CTA's and a warp's
// barriers as pthread barriers, shuffles through a warp's exchange slots.
// Only the barriers order anything, as on the device.
#pragma once
#include <pthread.h>
#include <sched.h>
#include <stdint.h>
#include <string.h>
#include <time.h>

#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>

#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
#define __restrict__

struct ulonglong2 {
  unsigned long long x, y;
};
inline ulonglong2 make_ulonglong2(unsigned long long x, unsigned long long y) { return {x, y}; }
struct Dim {
  unsigned x;
};
inline thread_local Dim threadIdx{0}, blockIdx{0};

namespace host {
struct Warp {
  pthread_barrier_t bar;
  unsigned long long slot[32];
};
struct Cta {
  pthread_barrier_t bar;
  std::vector<Warp> warps;
};
inline thread_local Cta* cta = nullptr;
inline Warp& warp() { return cta->warps[threadIdx.x / 32]; }

// Runs body() on `ctas` CTAs of `threads` threads.
template <class F>
void launch(unsigned ctas, unsigned threads, F body) {
  std::vector<Cta> grid(ctas);
  std::vector<std::thread> pool;
  for (unsigned b = 0; b < ctas; ++b) {
    pthread_barrier_init(&grid[b].bar, nullptr, threads);
    grid[b].warps.resize(threads / 32);
    for (Warp& w : grid[b].warps) pthread_barrier_init(&w.bar, nullptr, 32);
  }
  for (unsigned b = 0; b < ctas; ++b)
    for (unsigned t = 0; t < threads; ++t)
      pool.emplace_back([&, b, t] {
        cta = &grid[b];
        threadIdx.x = t;
        blockIdx.x = b;
        body();
      });
  for (std::thread& t : pool) t.join();
}

// The value `v` of lane `src` of the warp.
template <class T>
T exchange(T v, int src) {
  Warp& w = warp();
  unsigned long long q = 0;
  memcpy(&q, &v, sizeof(T));
  w.slot[threadIdx.x % 32] = q;
  pthread_barrier_wait(&w.bar);
  q = w.slot[src];
  pthread_barrier_wait(&w.bar);
  memcpy(&v, &q, sizeof(T));
  return v;
}
}  // namespace host

inline void __syncthreads() { pthread_barrier_wait(&host::cta->bar); }
inline void __syncwarp() { pthread_barrier_wait(&host::warp().bar); }
template <class T>
T __shfl_xor_sync(unsigned, T v, int mask) {
  return host::exchange(v, (int)(threadIdx.x % 32) ^ mask);
}
inline unsigned __reduce_max_sync(unsigned, unsigned v) {
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned b = __shfl_xor_sync(0u, v, o);
    v = v > b ? v : b;
  }
  return v;
}
inline bool __all_sync(unsigned, bool p) { return __reduce_max_sync(0u, p ? 0u : 1u) == 0u; }
inline int __double2hiint(double v) {
  unsigned long long q;
  memcpy(&q, &v, 8);
  return (int)(unsigned)(q >> 32);
}
inline int __double2loint(double v) {
  unsigned long long q;
  memcpy(&q, &v, 8);
  return (int)(unsigned)q;
}
inline double __hiloint2double(int hi, int lo) {
  const unsigned long long q = ((unsigned long long)(unsigned)hi << 32) | (unsigned)lo;
  double v;
  memcpy(&v, &q, 8);
  return v;
}
template <class T>
T __ldcg(const T* p) {
  return *p;
}
template <class T>
T __ldg(const T* p) {
  return *p;
}
inline int atomicExch(int* p, int v) { return __atomic_exchange_n(p, v, __ATOMIC_RELAXED); }
inline void __nanosleep(unsigned) { sched_yield(); }

namespace cup2d {
inline unsigned long long globaltimer_ns() {
  timespec t;
  clock_gettime(CLOCK_MONOTONIC, &t);
  return 1000000000ull * (unsigned long long)t.tv_sec + (unsigned long long)t.tv_nsec;
}
inline unsigned ld_acquire_u32(const unsigned* p) { return __atomic_load_n(p, __ATOMIC_ACQUIRE); }
inline int ld_volatile_s32(const int* p) { return __atomic_load_n(p, __ATOMIC_RELAXED); }
inline void red_release_add_u32(unsigned* p, unsigned v) { __atomic_fetch_add(p, v, __ATOMIC_RELEASE); }
}  // namespace cup2d
