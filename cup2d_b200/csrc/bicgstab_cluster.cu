// BiCGSTAB on one thread-block cluster: solves whose vectors fit the shared
// memory of up to 16 SMs.
//
// The grid solver (bicgstab.cu) spends a small solve on waiting: at 128 blocks
// an iteration took 19 us, 1-1.6 us in each of five barriers through L2 and 2-3
// us in passes that move a few KB each but begin with cold L2 loads.  Here the
// CTAs of one cluster hold everything an iteration touches: the Krylov vectors
// in lane-private slots, z in block order where the other CTAs read it through
// distributed shared memory, the solution's update, the addresses of the
// neighbour blocks and the explicit rows with the addresses of their operands
// (a cluster barrier's acquire drops L1, so tables left in global memory cost
// two dependent L2 reads in every SpMV).  Barriers are the cluster's hardware
// barrier, and a reduction posts each CTA's partial into every CTA's shared
// memory.
//
// The iteration, its scalars and its stop tests are those of the grid solver,
// with one rearrangement: the solution update x += alpha z + omega z2 is kept
// as y += alpha p + omega s (z = P^-1 p, z2 = P^-1 s and P^-1 is linear), and
// x = x0 + P^-1 y is formed when x is needed: at the end (FP64), at each
// true-residual replacement (mixed).  So z and z2 share one buffer and neither
// is read again after its SpMV.  y is FP64 in both forms.
//
// us an iteration, against the grid solver: FP64 128 blocks 17.1 -> 6.1, 449 17.1 ->
// 8.3, 899 17.5 -> 14.5; mixed 128 18.8 -> 7.8, 1,499 19.7 -> 17.0.  What is left of one
// at 128 blocks, in clocks when it took 6.7 us (13k): 4.8k in the two SpMV passes
// (dependent shared loads), some 4.5k in the three reductions, 2.4k in the block
// solves, 1.2k in the two barriers.
//
// Copies of the neighbours' blocks pushed ahead of each SpMV, so that no load
// left the CTA, measured no faster (their stores cost what the loads had).
//
// The CTAs of a cluster are co-resident and pass the same barriers.  All CTAs
// leave together: at the deadline, which is one of pass E's reduced quantities,
// or behind the next barrier when a reduction's bounded wait ran out in any of
// them (cluster_team.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "cluster_team.cuh"
#include "common.cuh"
#include "kernels.hpp"
#include "sine_solve.cuh"
#include "spmv.cuh"

namespace cup2d {

namespace {

constexpr int kMaxSweep = 64;  // mixed: longest FP32 sweep between true residuals

// Loads through the cluster's shared memory.  The conditional ones are
// predicated, not branched around: a chunk's and a row's loads then stay in
// flight together (with branches an SpMV pass of one chunk a warp took 4.3k
// clocks instead of 3.4k; with the long rows in shared memory too, 2.4k).
__device__ __forceinline__ double ld_cluster(uint32_t a, double) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ float ld_cluster(uint32_t a, float) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
// `other` where p does not hold
__device__ __forceinline__ double ld_cluster_if(bool p, uint32_t a, double other) {
  double v;
  asm volatile("{.reg .pred q; setp.ne.u32 q, %2, 0; mov.f64 %0, %3; @q ld.shared::cluster.f64 %0, [%1];}"
               : "=&d"(v)
               : "r"(a), "r"((unsigned)p), "d"(other));
  return v;
}
__device__ __forceinline__ float ld_cluster_if(bool p, uint32_t a, float other) {
  float v;
  asm volatile("{.reg .pred q; setp.ne.u32 q, %2, 0; mov.f32 %0, %3; @q ld.shared::cluster.f32 %0, [%1];}"
               : "=&f"(v)
               : "r"(a), "r"((unsigned)p), "f"(other));
  return v;
}
__device__ __forceinline__ void ld_cluster2_if(bool p, uint32_t a, double (&v)[2]) {
  asm volatile("{.reg .pred q; setp.ne.u32 q, %3, 0; @q ld.shared::cluster.v2.f64 {%0, %1}, [%2];}"
               : "+d"(v[0]), "+d"(v[1])
               : "r"(a), "r"((unsigned)p));
}
__device__ __forceinline__ void ld_cluster2_if(bool p, uint32_t a, float (&v)[2]) {
  asm volatile("{.reg .pred q; setp.ne.u32 q, %3, 0; @q ld.shared::cluster.v2.f32 {%0, %1}, [%2];}"
               : "+f"(v[0]), "+f"(v[1])
               : "r"(a), "r"((unsigned)p));
}
constexpr uint32_t kCodes = 1u;  // neighbour entries up to here: 0 wall, 1 coarse/fine face

__device__ __forceinline__ double prod(double a, double b) { return a * b; }
__device__ __forceinline__ double prod(float a, float b) { return (double)a * (double)b; }

// Fixed part of a CTA's shared memory.
struct ClHead {
  ClusterPosts posts;
  double sine[32][4];  // mixed: the FP64 block solve's constants per lane
  unsigned nlong;      // explicit rows longer than kRowWidth
};

constexpr int kSlotBytes = 512;  // one chunk of one vector: 16 bytes a lane
enum : int { kVr = 0, kVnu = 1, kVp = 2, kVrh = 3, kVt = 4, kPrivVecs = 5 };
// Explicit rows in shared memory: kRowWidth entries each (coarse/fine rows
// hold 7, 8 or 9), kLongWidth more for the first kLongRows longer ones (13:
// the corner cells between two such faces, some 1 % of the rows).
constexpr int kRowWidth = 9, kLongRows = 32, kLongWidth = 4;

struct ClRow {
  int cell, k0, len, ext;  // its cell, its first entry in the assembled rows, its entries; its place among the long rows or -1
};

// Offsets (bytes) of a CTA's arrays, the same in every CTA of the cluster.
// nbl: the most blocks a CTA has; rows: explicit rows kept in shared memory.
template <class T>
struct ClLayout {
  uint32_t z, y, slots, nbr, mask, addr, scratch, row, raddr, rval, laddr, lval, end;
  __host__ __device__ static uint32_t align(uint32_t v) { return (v + 15u) & ~15u; }
  __host__ __device__ ClLayout(int nb, int nbl, int rows) {
    const uint32_t nch = (uint32_t)(nbl + Frag<T>::CB - 1) / Frag<T>::CB, cells = nch * Frag<T>::CB * kBLEN;
    uint32_t o = align((uint32_t)sizeof(ClHead));
    z = o;
    o += cells * (uint32_t)sizeof(T);
    y = o;
    o += cells * 8u;
    slots = o;
    o += kPrivVecs * nch * kSlotBytes;
    nbr = o;
    o += (uint32_t)nbl * 16u;
    mask = o;
    o = align(o + (uint32_t)nbl * 8u);
    addr = o;
    o = align(o + (uint32_t)nb * 4u);
    scratch = o;
    o += kClWarps * 512u;
    row = o;
    o += (uint32_t)rows * (uint32_t)sizeof(ClRow);
    rval = align(o);
    o = rval + (uint32_t)rows * kRowWidth * (uint32_t)sizeof(T);
    raddr = align(o);
    const uint32_t longs = rows > 0 ? kLongRows * kLongWidth : 0;
    lval = align(raddr + (uint32_t)rows * kRowWidth * 4u);
    laddr = align(lval + longs * (uint32_t)sizeof(T));
    end = align(laddr + longs * 4u);
  }
};

extern __shared__ __align__(16) unsigned char g_cl_smem[];

// The lane-private vectors of a CTA.  Every pass hands the same cells to the
// same lane: chunk c (one FP64 block, two FP32 blocks) belongs to warp c mod
// (warps), and lane (g, t) of it holds row g, columns 2t and 2t+1 of each of its
// blocks, the fragment layout of the block solves, as 16 bytes of a slot.
template <class T>
struct Slots {
  static constexpr int CB = Frag<T>::CB, N = Frag<T>::N;
  T* base;
  int nch;     // chunks of this CTA
  int b0, b1;  // its blocks
  __device__ __forceinline__ T* slot(int v, int c) const { return base + (v * nch + c) * (kSlotBytes / (int)sizeof(T)); }
  __device__ __forceinline__ void ld(int v, int c, int lane, T (&a)[N]) const { lds16<N>(slot(v, c) + lane * N, a); }
  __device__ __forceinline__ void st(int v, int c, int lane, const T (&a)[N]) const { stv<N>(slot(v, c) + lane * N, a); }
  // the values whose bit of `skip` is clear
  __device__ __forceinline__ void st_masked(int v, int c, int lane, const T (&a)[N], unsigned skip) const {
    if (!__any_sync(kFull, skip != 0u)) {
      st(v, c, lane, a);
      return;
    }
    T* const p = slot(v, c) + lane * N;
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (!((skip >> j) & 1u)) p[j] = a[j];
  }
  // one cell of the CTA's blocks; an even cell and the next lie side by side
  __device__ __forceinline__ T& at(int v, int cell) const {
    const int lb = cell / kBLEN - b0;
    return slot(v, lb / CB)[((cell & (kBLEN - 1)) >> 1) * N + (lb % CB) * 2 + (cell & 1)];
  }
};

template <class T>
struct Cluster {
  static constexpr int CB = Frag<T>::CB, N = Frag<T>::N;
  const MeshView& M;
  ClusterTeam team;
  Slots<T> K;
  T* z;           // [nbl * 64], block order
  double* y;      // [nbl * 64]
  const uint4* nbr;                  // neighbour blocks' z, or a code
  const unsigned long long* mask;    // explicit rows of a block
  const uint32_t* addr;              // z of every block of the forest
  T* scratch;     // the warp's 512 bytes
  int r0, r1;     // explicit rows of the CTA's blocks, the first `kept` in shared memory:
  int kept;       // entry j of row i at [j * cap + i]
  int cap;
  const ClRow* row;
  const T* rval;
  const uint32_t* raddr;
  const T* lval;  // the long rows' further entries
  const uint32_t* laddr;

  __device__ __forceinline__ void st_z(int c, int lane, const T (&v)[N]) const {
#pragma unroll
    for (int j = 0; j < CB; ++j) {
      const T q[2] = {v[2 * j], v[2 * j + 1]};
      T* p = z + (c * CB + j) * kBLEN + 2 * lane;
      if constexpr (sizeof(T) == 8) *reinterpret_cast<double2*>(p) = make_double2(q[0], q[1]);
      else *reinterpret_cast<float2*>(p) = make_float2(q[0], q[1]);
    }
  }

  // A z: the stencil rows of the CTA's blocks, each chunk handed to
  // epi.chunk(c, lane, y, skip) (bit j of skip: value j is an explicit row's
  // or outside), and the explicit rows to epi.row(cell, y); summed left,
  // right, below, above as the grid solver does.  z must be visible.
  template <class Epi>
  __device__ __forceinline__ void spmv(Epi& epi) const {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    for (int c = w; c < K.nch; c += kClWarps) {
      T out[N];
      unsigned skip = 0;
#pragma unroll
      for (int j = 0; j < CB; ++j) {
        const int lb = c * CB + j;
        if (CB > 1 && K.b0 + lb >= K.b1) {
          out[2 * j] = out[2 * j + 1] = T(0);
          skip |= 3u << (2 * j);
          continue;
        }
        const T* zs = z + lb * kBLEN + 2 * lane;
        const uint4 nb = nbr[lb];
        const bool has_l = t > 0 || nb.x > kCodes, has_r = t < 3 || nb.y > kCodes;
        const bool has_d = g > 0 || nb.z > kCodes, has_u = g < 7 || nb.w > kCodes;
        T zc[2], dn[2], up[2];
        // inside the block from this CTA, across a face from the neighbour's;
        // a wall counts as zero and is left out of the diagonal
        T vl = ld_cluster_if(t == 0 && has_l, nb.x + (uint32_t)((g * 8 + 7) * sizeof(T)), T(0));
        T vr = ld_cluster_if(t == 3 && has_r, nb.y + (uint32_t)(g * 8 * sizeof(T)), T(0));
        lds_pair(zs, zc);
        lds_pair(zs - (g > 0 ? 8 : 0), dn);
        lds_pair(zs + (g < 7 ? 8 : 0), up);
        const T il = zs[t > 0 ? -1 : 0], ir = zs[t < 3 ? 2 : 0];
        if (!has_d) dn[0] = dn[1] = T(0);
        if (!has_u) up[0] = up[1] = T(0);
        ld_cluster2_if(g == 0 && has_d, nb.z + (uint32_t)((56 + 2 * t) * sizeof(T)), dn);
        ld_cluster2_if(g == 7 && has_u, nb.w + (uint32_t)(2 * t * sizeof(T)), up);
        if (t > 0) vl = il;
        if (t < 3) vr = ir;
        const T n = T(1 + (has_d ? 1 : 0) + (has_u ? 1 : 0));
        T a0 = vl + zc[1], a1 = zc[0] + vr;
        a0 = (a0 + dn[0]) + up[0];
        a1 = (a1 + dn[1]) + up[1];
        out[2 * j] = a0 - (has_l ? n + T(1) : n) * zc[0];
        out[2 * j + 1] = a1 - (has_r ? n + T(1) : n) * zc[1];
        skip |= ((unsigned)(mask[lb] >> (2 * lane)) & 3u) << (2 * j);
      }
      epi.chunk(c, lane, out, skip);
    }
    const T* __restrict__ vals = row_vals<T>(M);
    // from the last warp down: the first ones have one chunk more, or the only one
    for (int i = kClThreads - 1 - (int)threadIdx.x; i < r1 - r0; i += kClThreads) {
      T acc = T(0);
      int cell, k, k1;  // entries [k, k1) are left to the tables in global memory
      if (i < kept) {
        const ClRow rw = row[i];
        T x[kRowWidth];
#pragma unroll
        for (int j = 0; j < kRowWidth; ++j) x[j] = ld_cluster(raddr[j * cap + i], T(0));
#pragma unroll
        for (int j = 0; j < kRowWidth; ++j)
          acc = j < rw.len ? acc + rval[j * cap + i] * x[j] : acc;
        int done = kRowWidth;
        if (rw.ext >= 0) {
          const int n = min(rw.len - kRowWidth, kLongWidth);
          for (int j = 0; j < n; ++j)
            acc += lval[rw.ext * kLongWidth + j] * ld_cluster(laddr[rw.ext * kLongWidth + j], T(0));
          done += n;
        }
        cell = rw.cell;
        k = rw.k0 + done;
        k1 = rw.k0 + rw.len;
      } else {
        cell = __ldg(M.rowcell + r0 + i);
        k = __ldg(M.xptr + r0 + i);
        k1 = __ldg(M.xptr + r0 + i + 1);
      }
      for (; k < k1; ++k) {
        const int col = __ldg(M.xcol + k);
        acc += __ldg(vals + k) * ld_cluster(addr[col >> 6] + (uint32_t)((col & 63) * sizeof(T)), T(0));
      }
      epi.row(cell, acc);
    }
  }
};

// Epilogues of the SpMV passes (B: nu, (rhat, nu); D: t, (t, s), (t, t)).
template <class T>
struct ClRhNu {
  const Slots<T>& K;
  double acc;
  __device__ __forceinline__ void chunk(int c, int lane, const T (&y)[Frag<T>::N], unsigned skip) {
    T v[Frag<T>::N];
    K.ld(kVrh, c, lane, v);
    K.st_masked(kVnu, c, lane, y, skip);
#pragma unroll
    for (int j = 0; j < Frag<T>::N; ++j)
      if (!((skip >> j) & 1u)) acc += prod(v[j], y[j]);
  }
  __device__ __forceinline__ void row(int i, T y) {
    acc += prod(K.at(kVrh, i), y);
    K.at(kVnu, i) = y;
  }
};
template <class T>
struct ClTS {
  const Slots<T>& K;
  double ts, tt;
  __device__ __forceinline__ void chunk(int c, int lane, const T (&y)[Frag<T>::N], unsigned skip) {
    T v[Frag<T>::N];
    K.ld(kVr, c, lane, v);
    K.st_masked(kVt, c, lane, y, skip);
#pragma unroll
    for (int j = 0; j < Frag<T>::N; ++j)
      if (!((skip >> j) & 1u)) {
        ts += prod(y[j], v[j]);
        tt += prod(y[j], y[j]);
      }
  }
  __device__ __forceinline__ void row(int i, T y) {
    ts += prod(y, K.at(kVr, i));
    tt += prod(y, y);
    K.at(kVt, i) = y;
  }
};

// r = (b - mean_b) - A x in FP64 with x in global memory, rounded to T, and
// rhat = r when set_rh.  v: |A x|_inf, |r64|_inf, (rhat, r), |r|^2, |rhat|^2,
// |r|_inf of this thread.
template <class T>
struct ClResidual {
  const Slots<T>& K;
  const double* b;
  double mean_b;
  bool set_rh;
  double v[6];
  struct Pre {
    double b[2];
  };
  __device__ __forceinline__ Pre load(int i0) const {
    Pre p;
    ldv<2>(b + i0, p.b);
    return p;
  }
  __device__ __forceinline__ Pre load1(int i) const {
    Pre p{};
    p.b[0] = __ldg(b + i);
    return p;
  }
  __device__ __forceinline__ T acc(double y, double bi, T rhi) {
    const double r64 = (bi - mean_b) - y;
    const T rt = (T)r64;
    const T rhv = set_rh ? rt : rhi;
    v[0] = nanmax(v[0], fabs(y));
    v[1] = nanmax(v[1], fabs(r64));
    v[2] += prod(rhv, rt);
    v[3] += prod(rt, rt);
    v[4] += prod(rhv, rhv);
    v[5] = nanmax(v[5], fabs((double)rt));
    return rt;
  }
  __device__ __forceinline__ void vec(int i0, const double (&y)[2], const Pre& p) {
    T h[2] = {T(0), T(0)}, q[2];
    if (!set_rh) lds_pair(&K.at(kVrh, i0), h);
    q[0] = acc(y[0], p.b[0], h[0]);
    q[1] = acc(y[1], p.b[1], h[1]);
    stv<2>(&K.at(kVr, i0), q);
    if (set_rh) stv<2>(&K.at(kVrh, i0), q);
  }
  __device__ __forceinline__ void one(int i, double y, const Pre& p, int j) {
    const T q = acc(y, p.b[j], set_rh ? T(0) : K.at(kVrh, i));
    K.at(kVr, i) = q;
    if (set_rh) K.at(kVrh, i) = q;
  }
};

// x += P^-1 y over the CTA's blocks (global x, block order), the old x saved
// in xo first when it is the best iterate so far; y = 0 after it.
template <class T>
__device__ __forceinline__ void add_update(const Cluster<T>& C, const SineSolve<double>& sine, double* __restrict__ x,
                                           double* __restrict__ xo, bool save) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double* const m = reinterpret_cast<double*>(C.scratch);
  for (int lb = w; lb < C.K.b1 - C.K.b0; lb += kClWarps) {
    double* yp = C.y + lb * kBLEN + 2 * lane;
    const int i0 = (C.K.b0 + lb) * kBLEN + 2 * lane;
    double v[2], xv[2];
    ldv<2>(x + i0, xv);
    lds_pair(yp, v);
    if (save) stv<2>(xo + i0, xv);
    sine.apply(v, m, lane);
    xv[0] += v[0];
    xv[1] += v[1];
    stv<2>(x + i0, xv);
    *reinterpret_cast<double2*>(yp) = make_double2(0.0, 0.0);
  }
}

// One solve by one cluster.  T double: the reference's FP64 solve; float: the
// mixed form (FP32 Krylov vectors, FP64 solution and true residual).
template <class T>
__device__ void cluster_solve(const ClusterArgs<T>& S) {
  constexpr bool MIXED = sizeof(T) == 4;
  constexpr int CB = Frag<T>::CB, N = Frag<T>::N;
  const Problem<T>& V = S.prob;
  const SolveParams& sp = S.sp;
  const MeshView& M = V.M;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nb = (int)M.nb;
  const unsigned size = gridDim.x, rank = blockIdx.x;  // one cluster
  const unsigned long long deadline = globaltimer_ns() + S.timeout_ns;
  ClHead& head = *reinterpret_cast<ClHead*>(g_cl_smem);
  const ClLayout<T> L(nb, (nb + (int)size - 1) / (int)size, S.rows);
  const int b0 = share(nb, rank, size), b1 = share(nb, rank + 1, size), nbl = b1 - b0;
  Cluster<T> C{M,
               ClusterTeam{head.posts, rank, size, 0u, 0u},
               Slots<T>{reinterpret_cast<T*>(g_cl_smem + L.slots), (nbl + CB - 1) / CB, b0, b1},
               reinterpret_cast<T*>(g_cl_smem + L.z),
               reinterpret_cast<double*>(g_cl_smem + L.y),
               reinterpret_cast<const uint4*>(g_cl_smem + L.nbr),
               reinterpret_cast<const unsigned long long*>(g_cl_smem + L.mask),
               reinterpret_cast<const uint32_t*>(g_cl_smem + L.addr),
               reinterpret_cast<T*>(g_cl_smem + L.scratch + w * 512),
               __ldg(M.xbase + b0),
               __ldg(M.xbase + b1),
               0,
               S.rows,
               reinterpret_cast<const ClRow*>(g_cl_smem + L.row),
               reinterpret_cast<const T*>(g_cl_smem + L.rval),
               reinterpret_cast<const uint32_t*>(g_cl_smem + L.raddr),
               reinterpret_cast<const T*>(g_cl_smem + L.lval),
               reinterpret_cast<const uint32_t*>(g_cl_smem + L.laddr)};
  C.kept = min(C.r1 - C.r0, C.cap);
  const Slots<T>& K = C.K;
  const int nch = K.nch;
  SineSolve<T> pin;
  pin.init();
  // tables: every block's z address, the neighbours' addresses, the masks, the
  // explicit rows
  {
    uint32_t* addr = reinterpret_cast<uint32_t*>(g_cl_smem + L.addr);
    const uint32_t zbase = smem_u32(C.z);
    for (int b = threadIdx.x; b < nb; b += kClThreads) {
      const unsigned k = (unsigned)(((long long)(b + 1) * size - 1) / nb);
      addr[b] = cluster_addr(zbase + (uint32_t)((b - share(nb, k, size)) * kBLEN * sizeof(T)), k);
    }
    if (threadIdx.x == 0) head.nlong = 0u;
    head.posts.clear();
    if (MIXED && w == 0) {
      SineSolve<double> d;
      d.init();
      head.sine[lane][0] = d.s0;
      head.sine[lane][1] = d.s1;
      head.sine[lane][2] = d.d0;
      head.sine[lane][3] = d.d1;
    }
    for (int i = threadIdx.x; i < nch * CB * kBLEN; i += kClThreads) C.y[i] = 0.0;
    __syncthreads();
    uint32_t* nbr = reinterpret_cast<uint32_t*>(g_cl_smem + L.nbr);
    unsigned long long* mask = reinterpret_cast<unsigned long long*>(g_cl_smem + L.mask);
    for (int i = threadIdx.x; i < 4 * nbl; i += kClThreads) {
      const int code = __ldg(M.nbr + 4 * b0 + i);
      nbr[i] = code >= 0 ? addr[code] : code == kExplicit ? kCodes : 0u;
    }
    for (int i = threadIdx.x; i < nbl; i += kClThreads) mask[i] = __ldg(M.xmask + b0 + i);
    ClRow* row = reinterpret_cast<ClRow*>(g_cl_smem + L.row);
    T* rval = reinterpret_cast<T*>(g_cl_smem + L.rval);
    uint32_t* raddr = reinterpret_cast<uint32_t*>(g_cl_smem + L.raddr);
    T* lval = reinterpret_cast<T*>(g_cl_smem + L.lval);
    uint32_t* laddr = reinterpret_cast<uint32_t*>(g_cl_smem + L.laddr);
    const T* __restrict__ vals = row_vals<T>(M);
    for (int i = threadIdx.x; i < C.kept; i += kClThreads) {
      const int k0 = __ldg(M.xptr + C.r0 + i), len = __ldg(M.xptr + C.r0 + i + 1) - k0;
      int ext = -1;
      if (len > kRowWidth) {
        ext = (int)atomicAdd(&head.nlong, 1u);
        if (ext >= kLongRows) ext = -1;
        for (int j = 0; ext >= 0 && j < min(len - kRowWidth, kLongWidth); ++j) {
          const int col = __ldg(M.xcol + k0 + kRowWidth + j);
          laddr[ext * kLongWidth + j] = addr[col >> 6] + (uint32_t)((col & 63) * sizeof(T));
          lval[ext * kLongWidth + j] = __ldg(vals + k0 + kRowWidth + j);
        }
      }
      row[i] = ClRow{__ldg(M.rowcell + C.r0 + i), k0, len, ext};
      for (int j = 0; j < kRowWidth; ++j) {  // a short row is filled up with its first operand, times 0
        const int col = __ldg(M.xcol + k0 + (j < len ? j : 0));
        raddr[j * C.cap + i] = addr[col >> 6] + (uint32_t)((col & 63) * sizeof(T));
        rval[j * C.cap + i] = j < len ? __ldg(vals + k0 + j) : T(0);
      }
    }
  }
  C.team.sync();  // every CTA has started: its shared memory may be written
  // the FP64 block solve of x = x + P^-1 y
  auto sine64 = [&]() {
    SineSolve<double> d;
    if constexpr (MIXED) {
      d.s0 = head.sine[lane][0];
      d.s1 = head.sine[lane][1];
      d.d0 = head.sine[lane][2];
      d.d1 = head.sine[lane][3];
    } else {
      d = pin;
    }
    return d;
  };
  double* const row = reinterpret_cast<double*>(C.scratch);
  double mean_b = 0.0;
  bool lost = false;  // a wait ran out: the same for the cluster, which then leaves
  if constexpr (MIXED) {  // Neumann compatibility: project b to zero sum
    double v[1] = {0.0}, o[1];
    for (int blk = b0 + w; blk < b1; blk += kClWarps)
      v[0] += __ldg(V.b + blk * kBLEN + lane) + __ldg(V.b + blk * kBLEN + lane + 32);
    C.team.reduce(v, 0u, o);
    mean_b = o[0] / (double)(M.nb * kBLEN);
  }
  // r = b - A x (BiCGSTAB.cu:430-465)
  auto residual = [&](bool set_rh, double (&o)[6]) {
    ClResidual<T> epi{K, V.b, mean_b, set_rh, {0.0, 0.0, 0.0, 0.0, 0.0, 0.0}};
    spmv_range<double>(M, V.x, b0, b1, C.r0, C.r1, epi, row);
    C.team.reduce(epi.v, 0x23u, o);
  };
  double q[6];
  residual(true, q);
  const double norm_ax0 = q[0], err_init = q[1];
  double err_opt = err_init, err_true = err_init;
  double rho = q[2], nr = q[3], nrh = q[4];
  int restarts = 0, updates = 0, status = CUP2D_NOT_CONVERGED, k = 0;
  // FP64: y holds the best iterate (else xo does); mixed: x as of the last
  // replacement does
  bool best_here = true;
  bool expired = false;
  if (MIXED && (err_true <= sp.tol_abs || err_true == 0.0)) {
    status = CUP2D_OK;
  } else {
    const double eps = 1e-21;
    double rho_prev = 1.0, alpha = 1.0, omega = 1.0, beta;
    double alpha_omega = 1.0 / (1.0 + eps);
    bool zero_pnu = true;
    double rmax_since = sqrt(nr);
    int since = 0;
    for (; k < sp.max_iter; ++k) {
      // scalar step (BiCGSTAB.cu:471-509)
      const bool serious_breakdown = rho * rho < 1e-16 * nr * nrh;
      beta = (rho / (rho_prev + eps)) * alpha_omega;
      bool restart_now = false;
      if (serious_breakdown && sp.max_restarts > 0) {
        ++restarts;
        if (restarts >= sp.max_restarts) { status = CUP2D_BREAKDOWN_LIMIT; break; }
        restart_now = true;
        rho = nr;  // |rhat|^2 after rhat = r
        nrh = nr;
        zero_pnu = true;
        rho_prev = 1.0; alpha = 1.0; omega = 1.0;
        beta = (rho / (rho_prev + eps)) * (alpha / (omega + eps));
      }
      // pass A: p = r + beta (p - omega nu); z = P^-1 p
      {
        const T tb = (T)beta, to = (T)omega;
        for (int c = w; c < nch; c += kClWarps) {
          T pv[N];
          K.ld(kVr, c, lane, pv);
          if (restart_now) K.st(kVrh, c, lane, pv);
          if (!zero_pnu) {
            T pp[N], nn[N];
            K.ld(kVp, c, lane, pp);
            K.ld(kVnu, c, lane, nn);
#pragma unroll
            for (int j = 0; j < N; ++j) pv[j] = pv[j] + tb * (pp[j] - to * nn[j]);
          }
          K.st(kVp, c, lane, pv);
          pin.apply(pv, C.scratch, lane);
          C.st_z(c, lane, pv);
        }
        zero_pnu = false;
      }
      lost = !C.team.sync();
      if (lost) break;
      // pass B: nu = A z; (rhat, nu)
      {
        ClRhNu<T> epi{K, 0.0};
        C.spmv(epi);
        const double v[1] = {epi.acc};
        double o[1];
        C.team.reduce(v, 0u, o);
        alpha = rho / (o[0] + eps);
      }
      // pass C: s = r - alpha nu (in place of r); z = P^-1 s
      {
        const T ta = (T)alpha;
        for (int c = w; c < nch; c += kClWarps) {
          T sv[N], nn[N];
          K.ld(kVr, c, lane, sv);
          K.ld(kVnu, c, lane, nn);
#pragma unroll
          for (int j = 0; j < N; ++j) sv[j] = sv[j] - ta * nn[j];
          K.st(kVr, c, lane, sv);
          pin.apply(sv, C.scratch, lane);
          C.st_z(c, lane, sv);
        }
      }
      lost = !C.team.sync();
      if (lost) break;
      // pass D: t = A z; (t,s), (t,t)
      {
        ClTS<T> epi{K, 0.0, 0.0};
        C.spmv(epi);
        const double v[2] = {epi.ts, epi.tt};
        double o[2];
        C.team.reduce(v, 0u, o);
        omega = o[0] / (o[1] + eps);
      }
      // pass E: y += alpha p, y += omega s; r = s - omega t; norms; the
      // deadline.  FP64 saves the best iterate lazily: y still holds it.
      alpha_omega = alpha / (omega + eps);  // the division ahead of the wait
      double e[5];
      {
        const T to = (T)omega;
        double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        for (int c = w; c < nch; c += kClWarps) {
          const int nv = b1 - (b0 + c * CB);
          T pv[N], sv[N], tv[N], hv[N];
          double yv[N];
          K.ld(kVp, c, lane, pv);
          K.ld(kVr, c, lane, sv);
          K.ld(kVt, c, lane, tv);
          K.ld(kVrh, c, lane, hv);
#pragma unroll
          for (int j = 0; j < CB; ++j) {
            double a[2];
            lds_pair(C.y + (c * CB + j) * kBLEN + 2 * lane, a);
            yv[2 * j] = a[0];
            yv[2 * j + 1] = a[1];
          }
          if (!MIXED && best_here) stv<2>(V.xo + (b0 + c) * kBLEN + 2 * lane, *reinterpret_cast<double(*)[2]>(yv));
#pragma unroll
          for (int j = 0; j < N; ++j) {
            yv[j] = (yv[j] + alpha * (double)pv[j]) + omega * (double)sv[j];
            sv[j] = sv[j] - to * tv[j];
            if (CB == 1 || j < 2 * nv) {
              v[0] = nanmax(v[0], fabs((double)sv[j]));
              v[1] += prod(hv[j], sv[j]);
              v[2] += prod(sv[j], sv[j]);
              v[3] += prod(hv[j], hv[j]);
            }
          }
          K.st(kVr, c, lane, sv);
#pragma unroll
          for (int j = 0; j < CB; ++j)
            *reinterpret_cast<double2*>(C.y + (c * CB + j) * kBLEN + 2 * lane) =
                make_double2(yv[2 * j], yv[2 * j + 1]);
        }
        if (threadIdx.x == 0 && globaltimer_ns() > deadline) v[4] = 1.0;
        C.team.reduce(v, 0x11u, e);
      }
      if (e[4] != 0.0) {
        expired = true;
        break;
      }
      double error = e[0], rho_new = e[1];
      nr = e[2];
      nrh = e[3];
      if (!(error == error) || !(rho_new == rho_new)) {  // non-finite: stop, keep the best iterate
        if (!MIXED) best_here = false;
        ++k;
        break;
      }
      bool refreshed = false;
      if constexpr (MIXED) {
        rmax_since = fmax(rmax_since, sqrt(nr));
        ++since;
        const bool claims = (error <= sp.tol_abs) || (error / err_init <= sp.tol_rel);
        // replace the FP32 residual when it dropped by delta, claims
        // convergence, or a sweep stalls for kMaxSweep iterations
        if (claims || sqrt(nr) < sp.reliable_delta * rmax_since || since >= kMaxSweep) {
          since = 0;
          add_update(C, sine64(), V.x, V.xo, best_here);
          lost = !C.team.sync();  // x before its neighbours read it
          if (lost) break;
          residual(sp.reliable_restart != 0, q);
          ++updates;
          refreshed = true;
          err_true = q[1];
          rho_new = q[2];
          nr = q[3];
          nrh = q[4];
          error = q[5];
          rmax_since = sqrt(nr);
          best_here = err_true < err_opt;
          if (best_here) err_opt = err_true;
          if ((err_true <= sp.tol_abs) || (err_true / err_init <= sp.tol_rel)) {
            best_here = true;
            status = CUP2D_OK;
            ++k;
            break;
          }
        }
      } else if (error < err_opt) {  // convergence (BiCGSTAB.cu:571-600)
        err_opt = error;
        best_here = true;
        if ((error <= sp.tol_abs) || (error / err_init <= sp.tol_rel)) {
          status = CUP2D_OK;
          ++k;
          break;
        }
      } else {
        best_here = false;
      }
      if (MIXED && refreshed && sp.reliable_restart != 0) {
        // rhat = r was written with the true residual: fresh recurrences
        rho_prev = 1.0; alpha = 1.0; omega = 1.0;
        alpha_omega = 1.0 / (1.0 + eps);
        rho = rho_new;
        zero_pnu = true;
      } else {
        rho_prev = rho;
        rho = rho_new;
      }
    }
  }
  // every way out of the loop, but for a lost wait, passes one more barrier:
  // the wait that ran out may be the last reduction's
  if (lost || !C.team.sync() || expired) {
    if (threadIdx.x == 0) atomicExch(S.abort_flag, 1);
    return;
  }
  // the solution: FP64 x0 + P^-1 y of the best y, mixed the best x; then its
  // volume-weighted mean removed (ExpAMRSolver.cpp:383-415)
  double hx[2] = {0.0, 0.0};
  const SineSolve<double> sine = sine64();
  for (int lb = w; lb < nbl; lb += kClWarps) {
    const int i0 = (b0 + lb) * kBLEN + 2 * lane;
    double* yp = C.y + lb * kBLEN + 2 * lane;
    double v[2], xv[2];
    if constexpr (MIXED) {
      ldv<2>((best_here ? V.x : V.xo) + i0, xv);
    } else {
      if (best_here) lds_pair(yp, v);
      else ldv<2>(V.xo + i0, v);
      ldv<2>(V.x + i0, xv);
      sine.apply(v, row, lane);
      xv[0] += v[0];
      xv[1] += v[1];
    }
    *reinterpret_cast<double2*>(yp) = make_double2(xv[0], xv[1]);
    const double h = __ldg(M.hblk + b0 + lb);
    hx[0] += (xv[0] + xv[1]) * (h * h);
    hx[1] += 2.0 * (h * h);
  }
  double o[2] = {0.0, 1.0};
  if (sp.subtract_mean) C.team.reduce(hx, 0u, o);
  const double avg = sp.subtract_mean ? o[0] / o[1] : 0.0;
  for (int lb = w; lb < nbl; lb += kClWarps) {
    double xv[2];
    lds_pair(C.y + lb * kBLEN + 2 * lane, xv);
    if (sp.subtract_mean) {
      xv[0] -= avg;
      xv[1] -= avg;
    }
    stv<2>(V.x + (b0 + lb) * kBLEN + 2 * lane, xv);
  }
  if (rank == 0 && threadIdx.x == 0) {
    DevStats* s = V.stats;
    s->status = status;
    s->iterations = k;
    s->restarts = restarts;
    s->refinements = updates;
    s->err_init = err_init;
    s->err_opt = MIXED && status == CUP2D_OK ? err_true : err_opt;
    s->norm_ax0 = MIXED ? 0.0 : norm_ax0;
  }
  // no CTA leaves while another may read its shared memory
  if (!C.team.sync() && threadIdx.x == 0) atomicExch(S.abort_flag, 1);
}

__global__ void __launch_bounds__(kClThreads, 1) k_bicgstab64_cluster(const __grid_constant__ ClusterArgs<double> S) {
  cluster_solve<double>(S);
}
__global__ void __launch_bounds__(kClThreads, 1) k_bicgstab_mixed_cluster(const __grid_constant__ ClusterArgs<float> S) {
  cluster_solve<float>(S);
}

template <class T>
const void* cluster_fn() {
  if constexpr (sizeof(T) == 8) return (const void*)k_bicgstab64_cluster;
  else return (const void*)k_bicgstab_mixed_cluster;
}

// Shared memory of a CTA that keeps `rows` explicit rows.
template <class T>
size_t cluster_bytes(int64_t nb, int size, int rows) {
  if (nb > 1 << 16) return ~size_t(0);  // beyond any shared memory (and 32-bit offsets)
  return ClLayout<T>((int)nb, (int)((nb + size - 1) / size), rows).end;
}

// The most shared memory of a CTA, 0 where clusters of 16 such CTAs cannot run;
// asked once per device, and the kernels' attributes are set with it.
size_t cluster_limit(int device) {
  static std::atomic<int64_t> cache[64];
  if (device < 0 || device >= 64) return 0;
  int64_t v = cache[device].load(std::memory_order_acquire);
  if (v != 0) return v > 0 ? (size_t)v : 0;
  int optin = 0;
  bool ok = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) == cudaSuccess;
  for (const void* fn : {cluster_fn<double>(), cluster_fn<float>()}) {
    int active = 0;
    ok = ok && cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin) == cudaSuccess &&
         cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    if (!ok) break;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kMaxCluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kMaxCluster);
    cfg.blockDim = dim3(kClThreads);
    cfg.dynamicSmemBytes = (size_t)optin;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    ok = cudaOccupancyMaxActiveClusters(&active, fn, &cfg) == cudaSuccess && active > 0;
  }
  if (!ok) cudaGetLastError();
  cache[device].store(ok ? (int64_t)optin : -1, std::memory_order_release);
  return ok ? (size_t)optin : 0;
}

}  // namespace

// The cluster solver takes every forest whose vectors fit (FP64 about 940
// blocks, mixed 1,650), where it is still the faster one: us an iteration
// against the grid solver, FP64 899 blocks 14.5 / 17.5, mixed 1,601 18.2 / 19.6, and
// 10.6 / 17.9 on 575 blocks with 4,852 explicit rows.  Of the cluster sizes the
// smallest with at most 12 blocks a CTA: past it twice the SMs give at most 7 % (us
// in FP64 on 2 / 4 / 8 / 16 CTAs: 24 blocks 5.0 / 4.6 / 4.6 / 4.7, 48 blocks 6.5 / 5.0 / 4.7
// / 4.8, 96 blocks 8.9 / 6.6 / 5.0 / 4.8, 128 refined - / 9.4 / 7.3 / 6.1, 302 on 8 / 16
// 11.3 / 9.0; mixed 96 blocks 10.1 / 7.4 / 6.9 / 6.7), and several small solves share
// the device.
template <class T>
int cluster_size(int device, int64_t nb) {
  const size_t most = cluster_limit(device);
  if (most == 0) return 0;
  int size = 1;
  while (size < kMaxCluster && (nb > 12 * size || cluster_bytes<T>(nb, size, 0) > most)) size *= 2;
  return cluster_bytes<T>(nb, size, 0) <= most ? size : 0;
}
template int cluster_size<double>(int, int64_t);
template int cluster_size<float>(int, int64_t);

template <class T>
cudaError_t launch_bicgstab_cluster(ClusterArgs<T>& a, int size, cudaStream_t s) {
  int dev = 0;
  if (cudaError_t e = cudaGetDevice(&dev)) return e;
  const size_t most = cluster_limit(dev);
  const int64_t nb = a.prob.M.nb;
  if (cluster_bytes<T>(nb, size, 0) > most) return cudaErrorInvalidConfiguration;
  // explicit rows in shared memory: up to three times an even share (they lie
  // unevenly along the blocks' order), as far as it goes
  a.rows = (int)std::min<int64_t>(a.prob.M.R, 3 * ((a.prob.M.R + size - 1) / size) + 32);
  while (a.rows > 0 && cluster_bytes<T>(nb, size, a.rows) > most) a.rows -= std::min(a.rows, 32);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)size;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)size);
  cfg.blockDim = dim3(kClThreads);
  cfg.dynamicSmemBytes = cluster_bytes<T>(nb, size, a.rows);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void* args[] = {&a};
  return cudaLaunchKernelExC(&cfg, cluster_fn<T>(), args);
}
template cudaError_t launch_bicgstab_cluster<double>(ClusterArgs<double>&, int, cudaStream_t);
template cudaError_t launch_bicgstab_cluster<float>(ClusterArgs<float>&, int, cudaStream_t);

}  // namespace cup2d
