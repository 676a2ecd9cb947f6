// Forest adaptation on the device: the remesh step of a time-stepping run
// without a host forest.
//
// CUP2D adapts its forest every few steps (source/Operators/AdaptTheMesh.cpp:
// 80-110): it tags blocks by a refinement criterion, Cubism's MeshAdaptation
// refines/compresses them and restores the 2:1 balance, and the pressure
// solver re-assembles its operator (ExpAMRSolver.cpp:370-376).  Here the
// criterion is the benchmark's geometry (blocks meeting the band
// { p : | |p - c| - r | <= band } of a disk are refined to the finest level),
// and the whole forest is rebuilt on the device from it:
//
//   tag      level by level from the roots: a position exists when its parent
//            was refined; it is refined when it is above the finest level and
//            meets a band, else it is a leaf (one thread per position);
//   balance  every leaf at level l >= 2 looks at its 8 face and corner
//            neighbours; a covering leaf more than one level coarser is marked
//            and split into its 4 children; rounds of descending levels run
//            until a round marks nothing (the balanced refinement of a leaf
//            set is unique, so the order of the splits does not matter);
//   order    every leaf's Morton key (its finest-level corner, bits of i and j
//            interleaved) marks a dense key array, an exclusive scan of which
//            gives each leaf its position: the leaves in Morton order.
//
// One cooperative launch does all of it up to the ranks, with a grid barrier
// between the steps (about 1 us; some forty of them), a second writes the leaves
// once the host has sized their arrays.  As a launch per level and step it was
// some ninety launches and a host round trip per balance round.  Remesh of the
// 20,834-block forest (adaptation, assembly, read-back, transfer): 877 -> 560 us, 535
// with the eight neighbours of a leaf looked up together.
//
// The result is the forest the host generator builds for the same geometry
// (forest.cpp build_disk_forest: same geometric test with the same rounded
// operations, same balance rule, same order); the device assembly and the
// pressure transfer then take it from there.  States live in dense per-level
// byte arrays laid out like the assembly's leaf tables.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.hpp"

namespace cup2d {

namespace {

constexpr int kAdaptThreads = 1024;  // one CTA an SM

constexpr uint8_t kAbsent = 0, kLeaf = 1, kRefined = 2, kSplit = 3;  // kSplit: a leaf marked for splitting

__device__ __forceinline__ int64_t nx_at(const AdaptGeom& g, int l) { return (int64_t)g.bpdx << l; }
__device__ __forceinline__ int64_t ny_at(const AdaptGeom& g, int l) { return (int64_t)g.bpdy << l; }

// forest.cpp rect_meets_band with the host's rounding: separately rounded
// products and sums (no contraction into FMAs), correctly rounded sqrt.
__device__ __forceinline__ bool meets_band(double x0, double y0, double x1, double y1, double cx, double cy,
                                           double r, double band) {
  const double dx = fmax(fmax(__dadd_rn(x0, -cx), 0.0), __dadd_rn(cx, -x1));
  const double dy = fmax(fmax(__dadd_rn(y0, -cy), 0.0), __dadd_rn(cy, -y1));
  const double dmin = __dsqrt_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
  const double fx = fmax(fabs(__dadd_rn(x0, -cx)), fabs(__dadd_rn(x1, -cx)));
  const double fy = fmax(fabs(__dadd_rn(y0, -cy)), fabs(__dadd_rn(y1, -cy)));
  const double dmax = __dsqrt_rn(__dadd_rn(__dmul_rn(fx, fx), __dmul_rn(fy, fy)));
  return dmin <= __dadd_rn(r, band) && dmax >= __dadd_rn(r, -band);
}

// Positions of a level are shared out over the threads of the grid.  States
// that other CTAs wrote before a grid barrier are read from L2.
__device__ __forceinline__ int64_t grid_thread() { return blockIdx.x * (int64_t)blockDim.x + threadIdx.x; }
__device__ __forceinline__ int64_t grid_threads() { return (int64_t)gridDim.x * blockDim.x; }

__device__ __forceinline__ void adapt_tag(const AdaptGeom& g, const AdaptDisks& D, int l, uint8_t* state) {
  const int64_t nx = nx_at(g, l), n = nx * ny_at(g, l);
  // block size at this level: 8 * extent / (max(bpdx, bpdy) * 8 * 2^l), as forest.cpp cell_h
  const double h = __ddiv_rn(g.extent, __dmul_rn(__dmul_rn((double)max(g.bpdx, g.bpdy), 8.0), (double)(1ll << l)));
  const double bs = __dmul_rn(8.0, h);
  for (int64_t p = grid_thread(); p < n; p += grid_threads()) {
    const int64_t i = p % nx, j = p / nx;
    bool exists = l == 0;
    if (!exists) exists = __ldcg(state + g.off[l - 1] + (j >> 1) * nx_at(g, l - 1) + (i >> 1)) == kRefined;
    uint8_t st = kAbsent;
    if (exists) {
      bool refine = false;
      if (l < g.L - 1) {
        const double x0 = __dmul_rn((double)i, bs), y0 = __dmul_rn((double)j, bs);
        const double x1 = __dadd_rn(x0, bs), y1 = __dadd_rn(y0, bs);
        for (int k = 0; k < D.n && !refine; ++k)
          refine = meets_band(x0, y0, x1, y1, D.d[k][0], D.d[k][1], D.d[k][2], D.band);
      }
      st = refine ? kRefined : kLeaf;
    }
    state[g.off[l] + p] = st;
  }
}

// Level of the leaf covering position (l, i, j), or -1 when the position is
// refined (covered by finer leaves); a leaf marked for splitting still counts.
__device__ __forceinline__ int covering_level(const AdaptGeom& g, const uint8_t* state, int l, int64_t i, int64_t j) {
  for (int q = l; q >= 0; --q) {
    const int sh = l - q;
    const uint8_t s = __ldcg(state + g.off[q] + (j >> sh) * nx_at(g, q) + (i >> sh));
    if (s == kLeaf || s == kSplit) return q;
    if (s == kRefined) return -1;
  }
  return -1;
}

__device__ __forceinline__ void adapt_mark(const AdaptGeom& g, int l, uint8_t* state, int* changed) {
  const int64_t nx = nx_at(g, l), ny = ny_at(g, l), n = nx * ny;
  for (int64_t p = grid_thread(); p < n; p += grid_threads()) {
    const uint8_t s = __ldcg(state + g.off[l] + p);
    if (s != kLeaf && s != kSplit) continue;
    const int64_t i = p % nx, j = p / nx;
    // the 8 neighbours' states at this level and the next coarser one, loaded
    // together: nearly always the covering leaf is at one of the two, or finer
    uint8_t here[8], up[8];
    int64_t at_i[8], at_j[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int d = k < 4 ? k : k + 1;  // 3 x 3 without the middle
      int64_t ni = i + d % 3 - 1, nj = j + d / 3 - 1;
      bool in = true;
      if (ni < 0 || ni >= nx) {
        in = g.px;
        ni = ni < 0 ? ni + nx : ni - nx;
      }
      if (nj < 0 || nj >= ny) {
        in = in && g.py;
        nj = nj < 0 ? nj + ny : nj - ny;
      }
      at_i[k] = in ? ni : -1;
      at_j[k] = nj;
      here[k] = in ? __ldcg(state + g.off[l] + nj * nx + ni) : kLeaf;
      up[k] = in ? __ldcg(state + g.off[l - 1] + (nj >> 1) * nx_at(g, l - 1) + (ni >> 1)) : kLeaf;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (here[k] != kAbsent || up[k] != kAbsent) continue;
      const int64_t ni = at_i[k], nj = at_j[k];
      const int q = covering_level(g, state, l - 2, ni >> 2, nj >> 2);
      if (q >= 0) {
        const int sh = l - q;
        state[g.off[q] + (nj >> sh) * nx_at(g, q) + (ni >> sh)] = kSplit;
        *changed = 1;
      }
    }
  }
}

// Splits the marked leaves of level l into their four children.
__device__ __forceinline__ void adapt_split(const AdaptGeom& g, int l, uint8_t* state) {
  const int64_t nx = nx_at(g, l), n = nx * ny_at(g, l);
  for (int64_t p = grid_thread(); p < n; p += grid_threads()) {
    if (__ldcg(state + g.off[l] + p) != kSplit) continue;
    state[g.off[l] + p] = kRefined;
    const int64_t i = p % nx, j = p / nx, cnx = nx_at(g, l + 1);
    for (int c = 0; c < 4; ++c)
      state[g.off[l + 1] + (2 * j + (c >> 1)) * cnx + 2 * i + (c & 1)] = kLeaf;
  }
}

__device__ __forceinline__ uint64_t spread_bits(uint64_t v) {
  v &= 0xffffffffull;
  v = (v | (v << 16)) & 0x0000ffff0000ffffull;
  v = (v | (v << 8)) & 0x00ff00ff00ff00ffull;
  v = (v | (v << 4)) & 0x0f0f0f0f0f0f0f0full;
  v = (v | (v << 2)) & 0x3333333333333333ull;
  v = (v | (v << 1)) & 0x5555555555555555ull;
  return v;
}

__device__ __forceinline__ uint64_t leaf_key(const AdaptGeom& g, int l, int64_t i, int64_t j) {
  const int sh = g.L - 1 - l;
  return spread_bits((uint64_t)i << sh) | (spread_bits((uint64_t)j << sh) << 1);
}

// mark[key] = 1 for every leaf (the array is cleared before)
__device__ __forceinline__ void adapt_keys(const AdaptGeom& g, int l, const uint8_t* state, int32_t* mark) {
  const int64_t nx = nx_at(g, l), n = nx * ny_at(g, l);
  for (int64_t p = grid_thread(); p < n; p += grid_threads())
    if (__ldcg(state + g.off[l] + p) == kLeaf) mark[leaf_key(g, l, p % nx, p / nx)] = 1;
}

// rank[i] = marks before i over the dense key array, and their total: each CTA
// counts its share of the keys, and after the barrier every CTA adds the counts
// before its own.  Returns false if the barrier gave up.
__device__ __forceinline__ bool adapt_rank(Team& team, const int32_t* mark, int64_t K, int32_t* rank, int32_t* sums,
                                           int32_t* total) {
  __shared__ int warp_base[kAdaptThreads / 32];
  __shared__ int before;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t k0 = K * (int64_t)blockIdx.x / gridDim.x, k1 = K * (int64_t)(blockIdx.x + 1) / gridDim.x;
  int count = 0;
  for (int64_t t = k0; t < k1; t += kAdaptThreads) {
    const int64_t i = t + threadIdx.x;
    count += __syncthreads_count(i < k1 && __ldcg(mark + i) != 0);
  }
  if (threadIdx.x == 0) sums[blockIdx.x] = count;
  if (!team.sync(0)) return false;
  if (w == 0) {
    int a = 0;
    for (int c = lane; c < (int)blockIdx.x; c += 32) a += __ldcg(sums + c);
    a = warp_sum(a);
    if (lane == 0) before = a;
  }
  __syncthreads();
  int base = before;
  for (int64_t t = k0; t < k1; t += kAdaptThreads) {
    const int64_t i = t + threadIdx.x;
    const unsigned m = __ballot_sync(kFull, i < k1 && __ldcg(mark + i) != 0);
    if (lane == 0) warp_base[w] = __popc(m);
    __syncthreads();
    int b = base, all = 0;
    for (int q = 0; q < kAdaptThreads / 32; ++q) {
      if (q < w) b += warp_base[q];
      all += warp_base[q];
    }
    if (i < k1) rank[i] = b + __popc(m & ((1u << lane) - 1u));
    base += all;
    __syncthreads();
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total = base;
  return true;
}

__global__ void __launch_bounds__(kAdaptThreads, 1)
    k_adapt_build(const __grid_constant__ AdaptGeom g, const __grid_constant__ AdaptDisks D,
                  const __grid_constant__ AdaptScratch sc, int64_t K, unsigned long long timeout_ns) {
  __shared__ Team team;
  AdaptFlags& F = *sc.flags;
  if (threadIdx.x == 0) team.init(blockIdx.x, gridDim.x, &F.counter, nullptr, &F.abort_flag, timeout_ns, nullptr);
  __syncthreads();
  for (int64_t i = grid_thread(); i < K; i += grid_threads()) sc.mark[i] = 0;
  for (int l = 0; l < g.L; ++l) {
    adapt_tag(g, D, l, sc.state);
    if (!team.sync(0)) return;
  }
  // balance: rounds of descending levels until one marks nothing.  A round
  // carries the splits it causes down to the coarse levels, so two rounds
  // settle it in practice; the bound only guards the loop.
  bool settled = false;
  for (int round = 0; round < 4 * g.L + 4 && !settled; ++round) {
    for (int l = g.L - 1; l >= 2; --l) {
      adapt_mark(g, l, sc.state, &F.changed[round]);
      if (!team.sync(0)) return;
      // the marked leaves of every coarser level: their children are leaves,
      // not marked ones, so the levels do not affect each other
      for (int q = l - 2; q >= 0; --q) adapt_split(g, q, sc.state);
      if (!team.sync(0)) return;
    }
    settled = __ldcg(&F.changed[round]) == 0;  // written before the last barrier: the same for all
  }
  if (!settled) {
    if (blockIdx.x == 0 && threadIdx.x == 0) F.unsettled = 1;
    return;
  }
  for (int l = 0; l < g.L; ++l) adapt_keys(g, l, sc.state, sc.mark);
  if (!team.sync(0)) return;
  adapt_rank(team, sc.mark, K, sc.rank, sc.sums, &F.leaves);
}

__global__ void k_adapt_scatter(const __grid_constant__ AdaptGeom g, const __grid_constant__ AdaptScratch sc, int64_t nb,
                                int32_t* __restrict__ level, int32_t* __restrict__ bx, int32_t* __restrict__ by) {
  for (int l = 0; l < g.L; ++l) {
    const int64_t nx = nx_at(g, l), n = nx * ny_at(g, l);
    for (int64_t p = grid_thread(); p < n; p += grid_threads())
      if (sc.state[g.off[l] + p] == kLeaf) {
        const int64_t i = p % nx, j = p / nx;
        const int32_t b = sc.rank[leaf_key(g, l, i, j)];
        if (b < 0 || b >= nb) {  // cannot happen for a consistent scan; never write outside the arrays
          atomicExch(&sc.flags->scatter_err, 1);
          continue;
        }
        level[b] = l;
        bx[b] = (int32_t)i;
        by[b] = (int32_t)j;
      }
  }
}

}  // namespace

int64_t adapt_key_space(int bpdx, int bpdy, int level_max) {
  const int64_t finest = (int64_t)std::max(bpdx, bpdy) << (level_max - 1);
  int b = 0;
  while (((int64_t)1 << b) < finest) ++b;
  return (int64_t)1 << (2 * b);
}

int adapt_build(const AdaptGeom& g, const AdaptDisks& D, const AdaptScratch& sc, int64_t* nleaves,
                cudaStream_t s) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return CUP2D_CUDA_ERROR;
  const int64_t finest = ((int64_t)g.bpdx << (g.L - 1)) * ((int64_t)g.bpdy << (g.L - 1));
  const int grid =
      (int)std::max<int64_t>(1, std::min<int64_t>({(finest + kAdaptThreads - 1) / kAdaptThreads, sms, kAdaptMaxCtas}));
  int64_t K = adapt_key_space(g.bpdx, g.bpdy, g.L);
  unsigned long long timeout_ns = 20000000000ull;
  void* args[] = {const_cast<AdaptGeom*>(&g), const_cast<AdaptDisks*>(&D), const_cast<AdaptScratch*>(&sc), &K,
                  &timeout_ns};
  AdaptFlags f;
  if (cudaMemsetAsync(sc.flags, 0, sizeof(AdaptFlags), s) != cudaSuccess ||
      cudaLaunchCooperativeKernel((const void*)k_adapt_build, dim3(grid), dim3(kAdaptThreads), args, 0, s) !=
          cudaSuccess ||
      cudaMemcpyAsync(&f, sc.flags, sizeof(AdaptFlags), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess) {
    cudaGetLastError();
    return CUP2D_CUDA_ERROR;
  }
  if (f.abort_flag) return CUP2D_TIMEOUT;
  if (f.unsettled) return CUP2D_BAD_MESH;
  *nleaves = f.leaves;
  return CUP2D_OK;
}

int adapt_scatter(const AdaptGeom& g, const AdaptScratch& sc, int64_t nb, int32_t* level, int32_t* bx, int32_t* by,
                  cudaStream_t s) {
  const int64_t finest = ((int64_t)g.bpdx << (g.L - 1)) * ((int64_t)g.bpdy << (g.L - 1));
  k_adapt_scatter<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>((finest + 255) / 256, 4096)), 256, 0, s>>>(
      g, sc, nb, level, bx, by);
  int err = 0;
  if (cudaGetLastError() != cudaSuccess ||
      cudaMemcpyAsync(&err, &sc.flags->scatter_err, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return CUP2D_CUDA_ERROR;
  return err ? CUP2D_BAD_MESH : CUP2D_OK;
}

}  // namespace cup2d
