// Operator apply y = A x: the standalone SpMV of the library (the role of the
// reference's hd_cusparseSpMV on the assembled CSR, source/Poisson/BiCGSTAB.cu),
// built on the block structure instead of a CSR of the whole matrix.
//
// A warp takes two chunks at a time (a chunk: one FP64 block or two FP32
// blocks, 16 bytes of cells a lane) and holds the blocks' neighbours across
// their faces, one (FP64) or two (FP32) values a lane; the neighbour table's
// entries and the explicit-row masks are read one step ahead.  The cells and the
// face neighbours go out together, the neighbours inside the block come by
// shuffles; summed left, right, below, above and minus n z as the solver's SpMV
// does.  The rows on coarse/fine faces follow, CSR, one a thread.
//
// Bound by memory latency and the L2 reads of the halos' sectors; a CTA's warps
// take consecutive blocks, so that most neighbours hit L1.  us on 1.15 M blocks,
// one / two / four chunks a warp: FP64 267 / 237 / 230, FP32 182 / 125 / 142; on 0.1 M
// blocks 41 / 39 / 40 and 26 / 26 / 25.  Two for both types: four is 14 % behind in FP32,
// and in FP64 3 % ahead on the larger forest and 3 % behind on the smaller.  Tiles staged in shared memory by bulk copies
// with a CTA barrier a tile took 271 and 149, 46 and 31 (65 % of its time issuing).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "kernels.hpp"
#include "spmv.cuh"

namespace cup2d {

namespace {

constexpr int kApplyThreads = 256;
constexpr int kApplyWarps = kApplyThreads / 32;

template <class T>
__device__ __forceinline__ T from_lane(T v, int src) {
  return __shfl_sync(kFull, v, src & 31);
}
// The lane's cells of a chunk: 16 bytes.
__device__ __forceinline__ void ldg16(const double* p, double (&v)[2]) {
  const double2 a = __ldg(reinterpret_cast<const double2*>(p));
  v[0] = a.x; v[1] = a.y;
}
__device__ __forceinline__ void ldg16(const float* p, float (&v)[4]) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p));
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}

// A chunk (one FP64 block, two FP32 blocks) on its way: the lane's cells, its
// neighbours across the block's faces (absent ones 0), whether the faces of
// its block have same-level neighbours, and which of its cells are explicit rows'.
template <class T>
struct ApplyChunk {
  static constexpr int V = Lane<T>::V, LB = Lane<T>::LB, NG = 32 / LB;  // neighbours a lane holds
  T z[V], ghost[NG];
  unsigned present[NG], skip;
};

// The 5-point rows of the lane's cells.
template <class T>
__device__ __forceinline__ void chunk_rows(int lane, const Lane<T>& L, const ApplyChunk<T>& c, T (&out)[Lane<T>::V]) {
  constexpr int V = Lane<T>::V, LB = Lane<T>::LB, LR = Lane<T>::LR, NG = ApplyChunk<T>::NG;
  const int base = L.bl * LB;
  const bool first = L.ix0 == 0, last = L.ix0 + V == kBS, low = L.iy == 0, high = L.iy == kBS - 1;
  // the face neighbours: W, E by row and S, N by column (FP64: ghosts 0..31 of
  // the block one a lane; FP32: W, E the first, S, N the second of a lane)
  const unsigned px = c.present[0] >> base, py = NG == 1 ? c.present[0] >> 16 : c.present[NG - 1] >> base;
  const T hx = from_lane(c.ghost[0], base + (first ? 0 : 8) + L.iy);
  const T l = from_lane(c.z[V - 1], lane - 1), r = from_lane(c.z[0], lane + 1);
  const bool has_l = !first || (px & 1u), has_r = !last || (px >> 8 & 1u);
  const bool has_d = !low || (py & 1u), has_u = !high || (py >> 8 & 1u);
  const T n = T(2 + (has_d ? 1 : 0) + (has_u ? 1 : 0));
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const T hy = from_lane(c.ghost[NG - 1], base + (NG == 1 ? 16 : 0) + (low ? 0 : 8) + L.ix0 + j);
    const T d = from_lane(c.z[j], lane - LR), u = from_lane(c.z[j], lane + LR);
    T a = j > 0 ? c.z[j - 1] : first ? hx : l;
    a += j < V - 1 ? c.z[j + 1] : last ? hx : r;
    a = (a + (low ? hy : d)) + (high ? hy : u);
    T m = n;
    if (j == 0 && !has_l) m -= T(1);
    if (j == V - 1 && !has_r) m -= T(1);
    out[j] = a - m * c.z[j];
  }
}

constexpr int kChunks = 2;  // consecutive chunks a warp takes at a time

template <class T>
__global__ void __launch_bounds__(kApplyThreads) k_apply(MeshView M, const T* __restrict__ x, T* __restrict__ y) {
  constexpr int V = Lane<T>::V, LB = Lane<T>::LB, CB = Lane<T>::CB, NG = ApplyChunk<T>::NG, U = kChunks;
  const int lane = threadIdx.x & 31;
  const Lane<T> L(lane);
  const int nb = (int)M.nb, step = (int)gridDim.x * kApplyWarps * U * CB;
  int b = ((int)blockIdx.x * kApplyWarps + (int)(threadIdx.x >> 5)) * U * CB;
  int code[U][NG];
  unsigned long long mask[U];
  auto tables = [&](int start) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int blk = start + u * CB + L.bl;
      const bool in = blk < nb;
#pragma unroll
      for (int q = 0; q < NG; ++q) code[u][q] = in ? __ldg(M.nbr + 4 * blk + q * (LB / 8) + (L.sub >> 3)) : kWall;
      mask[u] = in ? __ldg(M.xmask + blk) : ~0ull;  // past the end: nothing is written
    }
  };
  tables(b);
  for (; b < nb; b += step) {
    ApplyChunk<T> c[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int blk = min(b + u * CB + L.bl, nb - 1);
      ldg16(x + (size_t)blk * kBLEN + L.cell0, c[u].z);
#pragma unroll
      for (int q = 0; q < NG; ++q) {
        // the neighbour's cell facing this lane's position along the face
        const int f = q * (LB / 8) + (L.sub >> 3), k = L.sub & 7;
        const int facing = f == 0 ? k * kBS + kBS - 1 : f == 1 ? k * kBS : f == 2 ? (kBS - 1) * kBS + k : k;
        c[u].ghost[q] = code[u][q] >= 0 ? __ldg(x + (size_t)code[u][q] * kBLEN + facing) : T(0);
        c[u].present[q] = __ballot_sync(kFull, code[u][q] >= 0);
      }
      c[u].skip = (unsigned)(mask[u] >> L.cell0) & ((1u << V) - 1u);
    }
    tables(b + step);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      T out[V];
      chunk_rows<T>(lane, L, c[u], out);
      T* const o = y + (size_t)(b + u * CB + L.bl) * kBLEN + L.cell0;
      if (c[u].skip == 0u) {
        stv<V>(o, out);
      } else {
#pragma unroll
        for (int j = 0; j < V; ++j)
          if (!((c[u].skip >> j) & 1u)) o[j] = out[j];
      }
    }
  }
  const int R = (int)M.R, all = (int)gridDim.x * kApplyThreads;
  constexpr int W = 9;  // the entries of nearly every row
  const T* __restrict__ vals = row_vals<T>(M);
  for (int r = (int)blockIdx.x * kApplyThreads + (int)threadIdx.x; r < R; r += all) {
    const int k0 = __ldg(M.xptr + r), k1 = __ldg(M.xptr + r + 1), cell = __ldg(M.rowcell + r);
    T acc = T(0);
    for (int q = k0; q < k1; q += W) {
      int col[W];
      T v[W];
#pragma unroll
      for (int j = 0; j < W; ++j) {
        col[j] = q + j < k1 ? __ldg(M.xcol + q + j) : 0;
        v[j] = q + j < k1 ? __ldg(vals + q + j) : T(0);
      }
#pragma unroll
      for (int j = 0; j < W; ++j)
        if (q + j < k1) acc += v[j] * __ldg(x + col[j]);
    }
    y[cell] = acc;
  }
}

template <class T>
cudaError_t launch_apply(const MeshView& M, const T* x, T* y, cudaStream_t s) {
  constexpr int kPerCta = kApplyWarps * kChunks * Lane<T>::CB;  // blocks a CTA takes at a time
  static std::atomic<int> cap[64];
  if (M.nb <= 0) return cudaSuccess;
  int dev = 0;
  if (cudaError_t e = cudaGetDevice(&dev)) return e;
  int c = dev >= 0 && dev < 64 ? cap[dev].load(std::memory_order_acquire) : 0;
  if (c == 0) {
    int sms = 0, per_sm = 0;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_apply<T>, kApplyThreads, 0);
    if (e != cudaSuccess) return e;
    c = std::max(1, sms * std::max(1, per_sm));
    if (dev >= 0 && dev < 64) cap[dev].store(c, std::memory_order_release);
  }
  const int64_t ctas = std::min<int64_t>((M.nb + kPerCta - 1) / kPerCta, c);
  k_apply<T><<<(unsigned)ctas, kApplyThreads, 0, s>>>(M, x, y);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_spmv64(const MeshView& M, const double* x, double* y, cudaStream_t s) {
  return launch_apply<double>(M, x, y, s);
}

cudaError_t launch_spmv32(const MeshView& M, const float* x, float* y, cudaStream_t s) {
  return launch_apply<float>(M, x, y, s);
}

}  // namespace cup2d
