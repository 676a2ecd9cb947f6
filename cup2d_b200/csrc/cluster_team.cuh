// The CTAs of one thread-block cluster that solve a problem together, and how
// they wait for one another (the grid's counterpart: Team in common.cuh).
//
// sync: the cluster's hardware barrier; what any thread of the cluster wrote
// before it, shared memory of any CTA included, is visible to every thread after it.
//
// reduce: sums (or maxima) of the CTAs' values, known to every thread on return.
// Each CTA writes its partial, tagged, into every CTA's shared memory and waits
// for the others' in its own: one way across (a cluster barrier behind the same
// stores took 740 clocks on 8 CTAs and 1020 on 16).  A CTA posts after all its
// warps have finished the pass, so what follows may overwrite what the pass read;
// it orders no other data (that takes sync).  Every CTA adds the partials in the
// same order, so all know the same bits and decide alike.
//
// The wait of a reduction is bounded, and a CTA whose wait ran out goes on with
// whatever it has: it posts, decides and arrives at barriers as the others do.
// Leaving at once would take its shared memory from under their posts and loads,
// and its decisions may now be others than theirs.  Instead it notes in every CTA
// the number of the next barrier, and all CTAs leave behind that one: sync
// returns false in every thread of the cluster or in none.  What this asks of
// the caller: behind a reduction that decides anything, every branch comes to a
// sync before another reduction.  A CTA that is ahead may lose a later wait while
// this one still looks at its note; a number above the barriers passed is that,
// and leaves the decision to that barrier.
#pragma once
#include "common.cuh"
#include "spmv.cuh"

namespace cup2d {

constexpr int kClThreads = 512;
constexpr int kClWarps = kClThreads / 32;
constexpr int kMaxCluster = 16;
// bound of a reduction's wait, some 0.3 s
#ifndef CUP2D_CLUSTER_POLLS
#define CUP2D_CLUSTER_POLLS (1u << 23)
#endif
constexpr unsigned kMaxPolls = CUP2D_CLUSTER_POLLS;

__device__ __forceinline__ uint32_t cluster_addr(uint32_t local, unsigned rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
  return a;
}
// Two 64-bit words; each is written and read whole.
__device__ __forceinline__ void st_cluster_words(uint32_t a, unsigned long long x, unsigned long long y) {
  asm volatile("st.relaxed.cluster.shared::cluster.v2.u64 [%0], {%1, %2};" ::"r"(a), "l"(x), "l"(y) : "memory");
}
__device__ __forceinline__ ulonglong2 ld_words(uint32_t a) {
  ulonglong2 v;
  asm volatile("ld.relaxed.cluster.shared::cta.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster_u32(uint32_t a, unsigned v) {
  asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned ld_cta_u32(uint32_t a) {
  unsigned v;
  asm volatile("ld.relaxed.cluster.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_barrier() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A CTA's part, at the same place in the shared memory of every CTA.
struct ClusterPosts {
  double wred[kClWarps][kRedMax];
  double out[2][kRedMax];                // the last two reductions' results
  // the CTAs' partials, posted by each into every CTA: {tag, low half} and
  // {tag, high half} of a double
  alignas(16) ulonglong2 post[2][kRedMax][kMaxCluster];
  unsigned lost;                         // the barrier behind which all leave, 0: none

  // All threads; a sync follows before the first reduction.
  __device__ __forceinline__ void clear() {
    if (threadIdx.x == 0) lost = 0u;
    for (int i = threadIdx.x; i < 2 * kRedMax * kMaxCluster; i += kClThreads)
      (&post[0][0][0])[i] = make_ulonglong2(0ull, 0ull);  // no tag
  }
};

struct ClusterTeam {
  ClusterPosts& S;
  unsigned rank, size;
  unsigned posts;     // reductions so far
  unsigned barriers;  // syncs so far

  // False (in every thread of the cluster): a wait ran out, leave.
  __device__ __forceinline__ bool sync() {
    cluster_barrier();
    ++barriers;
    return ld_cta_u32(smem_u32(&S.lost)) - 1u >= barriers;
  }

  // Sums (bit q of is_max: maxima) of v over the cluster's threads, in out.
  template <int NV>
  __device__ __forceinline__ void reduce(const double (&v)[NV], unsigned is_max, double (&out)[NV]) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    warp_partials<NV>(v, is_max, S.wred[w]);
    __syncthreads();
    const unsigned tag = ++posts, set = tag & 1u;
    if (w < NV) {
      const bool mx = (is_max >> w) & 1u;
      double r = S.wred[lane & (kClWarps - 1)][w];
#pragma unroll
      for (int o = kClWarps / 2; o > 0; o >>= 1) {
        const double b = __shfl_xor_sync(kFull, r, o);
        r = mx ? nanmax(r, b) : r + b;
      }
      const unsigned long long t = (unsigned long long)tag << 32;
      if (lane < (int)size)
        st_cluster_words(cluster_addr(smem_u32(&S.post[set][w][rank]), (unsigned)lane),
                         t | (unsigned)__double2loint(r), t | (unsigned)__double2hiint(r));
      ulonglong2 x = make_ulonglong2(0ull, 0ull);
      unsigned spins = 0;
      bool ready, all;
      do {
        if (lane < (int)size) x = ld_words(smem_u32(&S.post[set][w][lane]));
        ready = lane >= (int)size || ((unsigned)(x.x >> 32) == tag && (unsigned)(x.y >> 32) == tag);
        all = __all_sync(kFull, ready);
      } while (!all && ++spins < kMaxPolls);
      if (!all && lane < (int)size) st_cluster_u32(cluster_addr(smem_u32(&S.lost), (unsigned)lane), barriers + 1u);
      r = lane < (int)size ? __hiloint2double((int)(unsigned)x.y, (int)(unsigned)x.x) : 0.0;
#pragma unroll
      for (int o = kMaxCluster / 2; o > 0; o >>= 1) {
        const double b = __shfl_xor_sync(kFull, r, o);
        r = mx ? nanmax(r, b) : r + b;
      }
      if (lane == 0) S.out[set][w] = r;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NV; ++q) out[q] = S.out[set][q];
  }
};

}  // namespace cup2d
