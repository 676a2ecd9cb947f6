// Device-side building blocks shared by the Poisson kernels (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/cup2d_poisson.h"

namespace cup2d {

constexpr int kBS = 8;          // cells per block side (CUP2D _BS_)
constexpr int kBLEN = 64;       // cells per block
constexpr unsigned kFull = 0xffffffffu;

// Face codes stored per block and face in the mesh's neighbour table.
constexpr int32_t kWall = -1;      // non-periodic domain edge: no flux
constexpr int32_t kExplicit = -2;  // coarse/fine face: rows stored explicitly

// Device image of an assembled AMR Laplacian (block-structured).
//   nbr[4*b+f]  : same-level neighbour block across face f (0 Xm,1 Xp,2 Ym,3 Yp),
//                 or kWall / kExplicit
//   xmask[b]    : bit c set <=> row of cell c is stored explicitly
//   xbase[b]    : index of block b's first explicit row
//   xptr[R+1], xcol[nnz], xval[nnz] (+ xval32): explicit rows, CSR, columns
//                 ascending, values as the reference's row accumulation
struct MeshView {
  int64_t nb;
  const int32_t* __restrict__ nbr;
  const unsigned long long* __restrict__ xmask;
  const int32_t* __restrict__ xbase;
  const int32_t* __restrict__ xptr;
  const int32_t* __restrict__ xcol;
  const double* __restrict__ xval;
  const float* __restrict__ xval32;
  const double* __restrict__ hblk;     // cell size per block
  const int32_t* __restrict__ rowcell; // [R] cell index of each explicit row
  int64_t R;                           // explicit rows
};

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ int ld_volatile_s32(const int* p) {
  int v;
  asm volatile("ld.volatile.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void red_release_add_u32(unsigned* p, unsigned v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// max that propagates NaN (fmax drops it, which would let a blown-up
// residual read as converged)
__device__ __forceinline__ double nanmax(double a, double b) { return (a > b || a != a) ? a : b; }

// Maximum of non-negative (or NaN) values: their bits order like integers,
// NaN above all.
__device__ __forceinline__ double warp_max_nonneg(double v) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const unsigned mh = __reduce_max_sync(kFull, hi);
  const unsigned ml = __reduce_max_sync(kFull, hi == mh ? lo : 0u);
  return __hiloint2double((int)mh, (int)ml);
}

// The warp's partials of NV quantities into dst[0..NV): sums, and for bit q of
// is_max set (a literal at every use) maxima of non-negative values.  Two sums
// share their shuffles: a lane keeps one and hands the other over, so that
// four sums take 6 exchanges, not 20 (a shuffle costs the SM a clock for every
// warp: 40 a warp in the pass with four quantities).
template <int NV>
__device__ __forceinline__ void warp_partials(const double (&v)[NV], unsigned is_max, double* dst) {
  const int lane = threadIdx.x & 31;
  double s[NV + 3];
  int at[NV + 3], n = 0;
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    if ((is_max >> q) & 1u) {
      const double m = warp_max_nonneg(v[q]);
      if (lane == 0) dst[q] = m;
    } else {
      s[n] = v[q];
      at[n++] = q;
    }
  }
#pragma unroll
  for (int k = 0; k < NV; k += 4) {
    if (k >= n) break;
    const int m = n - k;  // sums left
    double a, b = 0.0;
    if (m == 1) {
      a = s[k] + __shfl_xor_sync(kFull, s[k], 16);
      a += __shfl_xor_sync(kFull, a, 8);
    } else {
      const bool up = (lane & 16) != 0;
      a = (up ? s[k + 1] : s[k]) + __shfl_xor_sync(kFull, up ? s[k] : s[k + 1], 16);
      if (m == 2) {
        a += __shfl_xor_sync(kFull, a, 8);
      } else {
        const double c3 = m > 3 ? s[k + 3] : 0.0;
        b = (up ? c3 : s[k + 2]) + __shfl_xor_sync(kFull, up ? s[k + 2] : c3, 16);
        const bool up8 = (lane & 8) != 0;
        a = (up8 ? b : a) + __shfl_xor_sync(kFull, up8 ? a : b, 8);
      }
    }
    a += __shfl_xor_sync(kFull, a, 4);
    a += __shfl_xor_sync(kFull, a, 2);
    a += __shfl_xor_sync(kFull, a, 1);
    // lanes 0, 16 hold sums k, k+1; lanes 8, 24 sums k+2, k+3
    if (lane == 0) dst[at[k]] = a;
    if (m > 1 && lane == 16) dst[at[k + 1]] = a;
    if (m > 2 && lane == 8) dst[at[k + 2]] = a;
    if (m > 3 && lane == 24) dst[at[k + 3]] = a;
  }
}

constexpr int kSolveThreads = 256;
constexpr int kWarps = kSolveThreads / 32;

// A team's reduction slots in global memory: two sets (a CTA may post the next
// reduction while another still reads the last) of kRedMax quantities, one
// double a CTA.
constexpr int kRedMax = 6;
constexpr int kRedWords = 2 * kRedMax;

// The CTAs that solve one problem together (the whole grid for a single
// solve, a group in a batch), and how they wait for one another.
//
// sync: a barrier built on a monotonically increasing arrival counter; the
// k-th barrier of a launch waits until the counter reaches k * size.  What
// any thread of the team wrote before it is visible to every thread after it
// (release by the arrival, acquire by the wait; the CTA barriers on both
// sides extend them to the CTA).
//
// reduce: sums (or maxima) of the CTAs' values, known to every thread on
// return.  Each CTA posts its partial, the team syncs, and every CTA adds the
// partials in the same fixed order: all take identical decisions and a result
// depends on the team size, never on timing.  All the CTA's warps read the
// partials (one or two loads a lane: one L2 round trip; a warp a quantity with
// ten loads a lane on 296 CTAs cost 2-3 us of each pass after a reduction).
// Measured, us an iteration with the counter barrier and the partials read this
// way, against fences around the counter and a warp a quantity: 20,834 blocks
// FP64 58.9 -> 48.5, mixed 48.4 -> 38.1; 1,500 blocks 26.7 -> 20.0.
// Polling tagged partials instead of the counter measured slower (1.6 -> 2.2-3.2
// us a wait: the polls of all CTAs queue on the few lines being written).
//
// Waits are bounded: past `deadline_ns` (globaltimer) or when another CTA
// raised `abort_flag`, the CTA raises the flag itself and the call returns
// false; callers then leave the kernel.  Every thread of the CTA must call
// them (they contain __syncthreads).
//
// Profiling (the device-side counterpart of CUP2D's DeviceProfiler regions,
// source/Utils/DeviceProfiler.cuh): when `prof` is set, thread 0 adds to
// prof[(cta*kProfPhases + phase)*2 + {0,1}] the ns spent computing the phase
// that ends at this barrier and the ns spent waiting in it.
constexpr int kProfPhases = 10;

// The state lives in shared memory and the waits are calls: inlined at every
// use they cost the passes their registers (up to 1.6 KB of spills a thread).
struct Team {
  unsigned rank, size;
  unsigned* counter;    // zeroed before the launch
  double* slots;        // [2][kRedMax][size]
  int* abort_flag;
  unsigned long long deadline_ns;
  unsigned long long* prof;
  unsigned long long last;  // when thread 0 left the previous barrier
  unsigned epoch;  // syncs passed so far by this CTA
  int flag;
  double wred[kWarps][kRedMax];  // the warps' partials
  double part[kWarps];
  double out[kRedMax];           // the last reduction's results

  // One thread; the caller synchronises the CTA before the first wait.
  __device__ __forceinline__ void init(unsigned rank_, unsigned size_, unsigned* counter_, double* slots_, int* abort_,
                                       unsigned long long timeout_ns, unsigned long long* prof_) {
    rank = rank_;
    size = size_;
    counter = counter_;
    slots = slots_;
    abort_flag = abort_;
    last = globaltimer_ns();
    deadline_ns = last + timeout_ns;
    prof = prof_;
    epoch = 0u;
  }

  // Whether to give up (called while spinning, and once per wait).
  __device__ __forceinline__ bool expired() const {
    if (ld_volatile_s32(abort_flag) == 0 && globaltimer_ns() <= deadline_ns) return false;
    atomicExch(abort_flag, 1);
    return true;
  }

  // Arrival and wait of one thread for the team.
  __device__ __forceinline__ void wait(int phase) {
    int ok = 1;
    const unsigned long long t_arrive = prof ? globaltimer_ns() : 0;
    red_release_add_u32(counter, 1u);
    const unsigned target = ++epoch * size;
    unsigned spins = 0;
    // the deadline bounds the whole launch: checked at every barrier (a
    // register read), the abort flag only while spinning
    if (globaltimer_ns() > deadline_ns) ok = !expired();
    while (ok && ld_acquire_u32(counter) < target) {
      if ((++spins & 63u) == 0 && expired()) ok = 0;
      if (spins > 256) __nanosleep(64);
    }
    if (prof) {
      const unsigned long long t_depart = globaltimer_ns();
      unsigned long long* p = prof + ((size_t)blockIdx.x * kProfPhases + phase) * 2;
      p[0] += t_arrive - last;
      p[1] += t_depart - t_arrive;
      last = t_depart;
    }
    flag = ok;
  }

  __device__ __noinline__ bool sync(int phase) {
    __syncthreads();
    if (threadIdx.x == 0) wait(phase);
    __syncthreads();
    return flag != 0;
  }

  // Posts the warps' partials (wred, nv quantities, bit q of is_max: a
  // maximum), syncs, and leaves the team's results in out.
  __device__ __noinline__ bool exchange(int nv, unsigned is_max, int phase) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned n = size;
    // read ahead of the barrier: behind it thread 0's wait advances epoch
    double* const set = slots + (size_t)(epoch & 1u) * kRedMax * n;
    __syncthreads();
    if (w == 0) {
      if (lane < nv) {
        double acc = wred[0][lane];
        for (int k = 1; k < kWarps; ++k)
          acc = ((is_max >> lane) & 1u) ? nanmax(acc, wred[k][lane]) : acc + wred[k][lane];
        set[lane * n + rank] = acc;
      }
      __syncwarp();
      if (lane == 0) wait(phase);
    }
    __syncthreads();
    if (flag == 0) return false;
    // `per` warps read one quantity
    const int per = nv == 1 ? 8 : nv == 2 ? 4 : nv <= 4 ? 2 : 1;
    const int q = w / per, sub = w % per;
    if (q < nv) {
      const bool mx = (is_max >> q) & 1u;
      const double* src = set + q * n;
      const unsigned step = per * 32;
      double acc = 0.0;
      for (unsigned j0 = sub * 32 + lane; j0 < n; j0 += 5 * step) {
        double x[5];
#pragma unroll
        for (int u = 0; u < 5; ++u) x[u] = j0 + u * step < n ? __ldcg(src + j0 + u * step) : 0.0;
#pragma unroll
        for (int u = 0; u < 5; ++u) acc = mx ? nanmax(acc, x[u]) : acc + x[u];
      }
      __syncwarp();
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double b = __shfl_xor_sync(kFull, acc, o);
        acc = mx ? nanmax(acc, b) : acc + b;
      }
      if (lane == 0) part[w] = acc;
    }
    __syncthreads();
    if (threadIdx.x < nv) {
      const int k = threadIdx.x;
      double acc = part[k * per];
      for (int u = 1; u < per; ++u) acc = ((is_max >> k) & 1u) ? nanmax(acc, part[k * per + u]) : acc + part[k * per + u];
      out[k] = acc;
    }
    __syncthreads();
    return true;
  }

  // Sums (bit q of is_max: maxima) of v over the threads of the team; the
  // results are in out until the next reduction.
  template <int NV>
  __device__ __forceinline__ bool reduce(const double (&v)[NV], unsigned is_max, int phase) {
    static_assert(NV <= kRedMax, "reduction slots");
    warp_partials<NV>(v, is_max, wred[threadIdx.x >> 5]);
    return exchange(NV, is_max, phase);
  }
};

__host__ __device__ __forceinline__ int64_t imin64(int64_t a, int64_t b) { return a < b ? a : b; }

// Start of part k of n equal parts of [0, total): 64-bit product, 32-bit
// result (cell and block indices of one problem fit in 31 bits).
__device__ __forceinline__ int share(long long total, unsigned k, unsigned n) {
  return (int)(total * (long long)k / (long long)n);
}

template <class T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

template <class T>
__device__ __forceinline__ T warp_max(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(kFull, v, o));
  return v;
}

// FP64 tensor-core MMA, D(8x8) += A(8x4, row) * B(4x8, col).
// Lane l holds A[l/4][l%4], B[l%4][l/4], and C[l/4][2*(l%4) + {0,1}].
__device__ __forceinline__ void dmma_884(double& d0, double& d1, double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

}  // namespace cup2d
