// z = P^-1 p per 8x8 block by fast diagonalisation: the block-Jacobi
// preconditioner of the solve (the role of the reference's
// cublasDgemm(T, N, 64, Nblocks, 64) with P_inv, source/Poisson/BiCGSTAB.cu:520,545).
//
// P is the negated 5-point Laplacian of one 8x8 block with zero values
// outside (ExpAMRSolver.cpp:25-99), T x I + I x T with T = tridiag(-1, 2, -1).
// T is diagonalised by the orthonormal sine matrix S (symmetric, S S = I),
// S[j][k] = sqrt(2/9) sin(pi (j+1)(k+1) / 9), lambda_k = 4 sin^2(pi (k+1) / 18),
// so on the block's values X (row iy, column ix)
//   P^-1 X = -S (D o (S X S)) S,   D[i][j] = 1 / (lambda_i + lambda_j):
// four 8x8x8 products instead of one 64x64 matrix-vector product (1/8 of the
// multiply-adds).
//
// One warp handles a chunk in the tensor cores' own fragment layout: lane
// (g, t) = (lane / 4, lane % 4) holds cells (row g, columns 2t, 2t+1) of the
// block (FP64) or of each of two blocks (FP32).  A product with S from the
// right then needs no data movement: the k index of an MMA may run over the
// columns in any order, so the even columns form one half of k and the odd
// ones the other (A[g][t] = X[g][2t], B[t][n] = S[2t][n], then 2t+1), and the
// accumulators come out in the same layout.  Products from the left are
// products from the right of the transpose: two warp-local 8x8 transposes
// through 512 bytes of shared memory, swizzled so that neither the stores nor
// the loads meet a bank conflict.
//
// Bound by the vectors' traffic (L2 or HBM), not by the arithmetic (FP64: 8
// DMMAs a block, 32 clocks of an SM's FP64 pipe).  Measured on the 20,834-block
// forest (1.33 M cells, vectors in L2), us per pass, dense form -> this one:
// FP64 A 13.6 -> 10.6, C 12.0 -> 6.9; mixed A 10.5 -> 8.8, C 8.8 -> 6.8.  512
// uneven problems in one mixed launch: 659 -> 604 ms; 90 in FP64: 126 -> 115 ms.
//
// Nothing is shared between warps: no CTA barrier, no P^-1 in shared memory
// (the dense form kept 32 KB of it per CTA and re-read 64 KB of fragments per
// 4 KB tile), and z comes out in the lanes that hold p.
//
// FP32: every product is split into TF32 terms, x = xh + xl, S = Sh + Sl,
// X S = Xh Sh + Xl Sh + Xh Sl accumulated in FP32.
#pragma once
#include "common.cuh"
#include "spmv.cuh"

namespace cup2d {

// The cells of a chunk one lane holds: rows cell0 = 8 g + 2 t, two columns,
// of CB consecutive blocks.
template <class T>
struct Frag {
  static constexpr int CB = sizeof(T) == 8 ? 1 : 2;  // blocks per chunk (= Lane<T>::CB)
  static constexpr int N = 2 * CB;                   // values per lane
  static __device__ __forceinline__ int cell0(int lane) { return 2 * lane; }
};

// The lane's cells of a chunk from block blk (nv of its CB blocks exist; the
// others read 0 and are not written).
template <class T>
__device__ __forceinline__ void ld_frag(const T* v, int blk, int nv, int lane, T (&a)[Frag<T>::N]) {
#pragma unroll
  for (int j = 0; j < Frag<T>::CB; ++j) {
    T q[2] = {T(0), T(0)};
    if (j < nv) ldv<2>(v + (blk + j) * kBLEN + Frag<T>::cell0(lane), q);
    a[2 * j] = q[0];
    a[2 * j + 1] = q[1];
  }
}
template <class T>
__device__ __forceinline__ void st_frag(T* v, int blk, int nv, int lane, const T (&a)[Frag<T>::N]) {
#pragma unroll
  for (int j = 0; j < Frag<T>::CB; ++j) {
    const T q[2] = {a[2 * j], a[2 * j + 1]};
    if (j < nv) stv<2>(v + (blk + j) * kBLEN + Frag<T>::cell0(lane), q);
  }
}

__device__ __forceinline__ uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ double sine_entry(int j, int k) {
  return sqrt(2.0 / 9.0) * sinpi((double)(((j + 1) * (k + 1)) % 18) / 9.0);
}
__device__ __forceinline__ double sine_scale(int i, int j) {
  const double a = sinpi((double)(i + 1) / 18.0), b = sinpi((double)(j + 1) / 18.0);
  return -1.0 / (4.0 * a * a + 4.0 * b * b);
}

template <class T>
struct SineSolve;

template <>
struct SineSolve<double> {
  double s0, s1;  // S[2t][g], S[2t+1][g]
  double d0, d1;  // -D[g][2t], -D[g][2t+1]
  __device__ __forceinline__ void init() {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    s0 = sine_entry(2 * t, g);
    s1 = sine_entry(2 * t + 1, g);
    d0 = sine_scale(g, 2 * t);
    d1 = sine_scale(g, 2 * t + 1);
  }
  // v <- v S (rows of the warp's 8x8 block)
  __device__ __forceinline__ void times_s(double (&v)[2]) const {
    double c0 = 0.0, c1 = 0.0;
    dmma_884(c0, c1, v[0], s0);
    dmma_884(c0, c1, v[1], s1);
    v[0] = c0;
    v[1] = c1;
  }
  // Transpose of the block through `m` (64 doubles).  16-byte pieces: row r
  // holds pieces 0..3, two rows fill a 128-byte line; the piece's place in
  // the line is flipped by the row pair so that the column reads of a half
  // warp (4 row pairs x 2 pieces) hit eight different places.
  __device__ __forceinline__ static int place(int r, int piece) {
    const int t = r >> 1;
    return (t << 4) + ((((((r & 1) << 2) | piece) ^ ((t & 1) << 2)) ^ ((t >> 1) << 1)) << 1);
  }
  __device__ __forceinline__ static void transpose(double (&v)[2], double* m, int lane) {
    const int g = lane >> 2, t = lane & 3;
    __syncwarp();
    *reinterpret_cast<double2*>(m + place(g, t)) = make_double2(v[0], v[1]);
    __syncwarp();
    v[0] = m[place(2 * t, g >> 1) + (g & 1)];
    v[1] = m[place(2 * t + 1, g >> 1) + (g & 1)];
  }
  __device__ __forceinline__ void apply(double (&v)[2], double* m, int lane) const {
    times_s(v);
    transpose(v, m, lane);
    times_s(v);
    v[0] *= d0;  // D is symmetric: the same entries for the transpose
    v[1] *= d1;
    times_s(v);
    transpose(v, m, lane);
    times_s(v);
  }
};

template <>
struct SineSolve<float> {
  uint32_t h0, h1, l0, l1;  // TF32 split of S[2t][g], S[2t+1][g]
  float d0, d1;
  __device__ __forceinline__ void init() {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const double a = sine_entry(2 * t, g), b = sine_entry(2 * t + 1, g);
    h0 = to_tf32((float)a);
    l0 = to_tf32((float)(a - (double)__uint_as_float(h0)));
    h1 = to_tf32((float)b);
    l1 = to_tf32((float)(b - (double)__uint_as_float(h1)));
    d0 = (float)sine_scale(g, 2 * t);
    d1 = (float)sine_scale(g, 2 * t + 1);
  }
  // v = {block 0: columns 2t, 2t+1; block 1: the same}: MMA rows g are block
  // 0's, rows g + 8 block 1's
  __device__ __forceinline__ void times_s(float (&v)[4]) const {
    const float x[4] = {v[0], v[2], v[1], v[3]};
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      hi[k] = to_tf32(x[k]);
      lo[k] = to_tf32(x[k] - __uint_as_float(hi[k]));
    }
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    mma_tf32(acc, hi, l0, l1);
    mma_tf32(acc, lo, h0, h1);
    mma_tf32(acc, hi, h0, h1);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = acc[k];
  }
  // Transposes of both blocks through `m` (128 floats): rows of 8 words, four
  // to a 128-byte line, the second line's rows shifted by one place so that
  // the column reads (rows 2t or 2t+1, t = 0..3) fall in four different
  // quarters of the banks.
  __device__ __forceinline__ static int place(int r) { return ((r >> 2) << 5) + (((r & 3) ^ (r >> 2)) << 3); }
  __device__ __forceinline__ static void transpose(float (&v)[4], float* m, int lane) {
    const int g = lane >> 2, t = lane & 3;
    __syncwarp();
    *reinterpret_cast<float2*>(m + place(g) + 2 * t) = make_float2(v[0], v[1]);
    *reinterpret_cast<float2*>(m + 64 + place(g) + 2 * t) = make_float2(v[2], v[3]);
    __syncwarp();
    v[0] = m[place(2 * t) + g];
    v[1] = m[place(2 * t + 1) + g];
    v[2] = m[64 + place(2 * t) + g];
    v[3] = m[64 + place(2 * t + 1) + g];
  }
  __device__ __forceinline__ void apply(float (&v)[4], float* m, int lane) const {
    times_s(v);
    transpose(v, m, lane);
    times_s(v);
    v[0] *= d0;
    v[1] *= d1;
    v[2] *= d0;
    v[3] *= d1;
    times_s(v);
    transpose(v, m, lane);
    times_s(v);
  }
};

}  // namespace cup2d
