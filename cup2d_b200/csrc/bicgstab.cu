// BiCGSTAB with the 64x64 block-Jacobi preconditioner, one persistent launch
// per solve.
//
//   k_bicgstab64     plain FP64: the drop-in form of BiCGSTABSolver::main
//                    (source/Poisson/BiCGSTAB.cu:412-620)
//   k_bicgstab_mixed FP32 Krylov vectors and FP32 P^-1; FP64 solution
//                    update, FP64 true-residual replacement ("reliable
//                    updates") and FP64 convergence test
// P^-1 is applied as sine transforms in registers (sine_solve.cuh).
//
// The reference runs each iteration as ~25 library launches (cuSPARSE COO
// SpMV, cuBLAS dot/nrm2/axpy/scal/Idamax/Dgemm), 8 one-thread scalar kernels
// and 4 host round-trips.  Here one cooperative kernel runs the whole solve.
// Each CTA owns an equal contiguous range of blocks, and an equal share of
// the explicit (coarse/fine) rows for the SpMVs; an iteration is five fused
// passes over them, separated by bounded grid barriers:
//
//   A  p = r + beta (p - omega nu);  z = P^-1 p          (R r,p,nu  W p,z)
//   B  nu = A z;  (rhat, nu)                             (R z,rhat  W nu)
//   C  s = r - alpha nu;  z2 = P^-1 s                    (R r,nu    W s,z2)
//   D  t = A z2;  (t,s), (t,t)                           (R z2,s    W t)
//   E  x += alpha z, x += omega z2;  r = s - omega t;
//      |r|_inf, (rhat,r), |r|^2, |rhat|^2                (R x,z,z2,s,t,rhat W x,r)
//
// The two x updates of the reference (alpha z after the first half step,
// omega z2 after the second) are applied in that order in pass E, which
// gives the same values while touching x once per iteration.
//
// Scalar recurrences, the breakdown/restart rule (rho^2 < 1e-16|r|^2|rhat|^2),
// best-iterate tracking and the L-inf stopping test follow the reference.
// Every CTA reduces the per-CTA partials in the same fixed order (FP64), so
// all CTAs take identical decisions and results are bitwise reproducible for
// a given grid.  The best iterate is copied lazily: pass E of the next
// iteration stores the old x when the previous iterate was the best so far.
//
// Mixed form.  A correction accumulated in FP32 loses eps32*kappa of the
// residual (kappa ~ 1e5..1e7 on these meshes), so restarted FP32 inner
// solves cannot refine.  Instead x stays FP64 and is updated in pass E from
// the FP32 z and z2; only the Krylov vectors (r, rhat, p, nu, t, z, z2) are
// FP32.  When the FP32 residual has dropped by `reliable_delta` since its
// last replacement, claims convergence, or a sweep stalls, it is replaced by
// the true residual b - A x computed in FP64 (with b projected to zero sum,
// the Neumann compatibility condition); by default the recurrences restart
// from it (rhat = r, p = nu = 0), which FP32 needs here: on the large
// meshes the unrestarted FP32 recurrences diverge.  Convergence is declared
// only on the true FP64 residual, and the best iterate (returned when the
// solve stops unconverged) is the refreshed x with the lowest true residual.
#include <cuda_runtime.h>

#include <atomic>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.hpp"
#include "sine_solve.cuh"
#include "spmv.cuh"

namespace cup2d {

namespace {

constexpr int kMaxSweep = 64;  // mixed: longest FP32 sweep between true residuals

// Shared memory of the solve kernels, per precision T of the Krylov vectors:
// per warp one ring of the staged SpMV, which also serves as the scratch of
// the block solves' transposes and of the register-path SpMV, and the
// reduction scratch.
template <class T>
struct Smem {
  SpmvStage<T> stage[kWarps];
  Team team;
  int slot;  // batch: the problem the team works on
};

template <class T>
__device__ __forceinline__ SpmvStage<T>& spmv_stage(Smem<T>& sm) { return sm.stage[threadIdx.x >> 5]; }

// The warp's scratch of kBLEN doubles (its ring is idle outside passes B and
// D): the transposes of passes A and C, the block row of the FP64 SpMV.
template <class T>
__device__ __forceinline__ T* warp_scratch(Smem<T>& sm) { return spmv_stage(sm).z[0]; }
template <class T>
__device__ __forceinline__ double* spmv_row(Smem<T>& sm) { return reinterpret_cast<double*>(spmv_stage(sm).z[0]); }

// ----------------------------------------------------- iteration core -----

// bMeanConstraint (BiCGSTAB.cu:393-410, ExpAMRSolver.cpp:251-256, 340-346):
// the SpMV's row `mean_row` is replaced by sum_i h_i^2 v_i over the operand v
// and the right-hand side reads 0 there.  Each CTA adds the h^2-weighted sum
// of its own blocks of v (this thread's share).
template <class T>
__device__ __forceinline__ double hsum_part(const MeshView& M, const T* __restrict__ v, int b0, int b1) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double a = 0.0;
  for (int blk = b0 + w; blk < b1; blk += kWarps) {
    const double hb = __ldg(M.hblk + blk);
    const int o = blk * kBLEN;
    a += ((double)__ldcg(v + o + lane) + (double)__ldcg(v + o + lane + 32)) * (hb * hb);
  }
  return a;
}

__device__ __forceinline__ bool owns_row(int row, int b0, int b1) { return row >= b0 * kBLEN && row < b1 * kBLEN; }

// Whether this CTA's SpMV computes row `row`: a cell on a coarse/fine face
// (its block's explicit mask bit set; possible for the corner cell across a
// periodic edge) is an explicit row, computed by the CTA whose row range
// [r0, r1) holds it; any other cell by the owner of its block.
__device__ __forceinline__ bool computes_row(const MeshView& M, int row, int b0, int b1, int r0, int r1) {
  const int blk = row / kBLEN, c = row % kBLEN;
  const unsigned long long m = __ldg(M.xmask + blk);
  if ((m >> c) & 1ull) {
    const int xr = __ldg(M.xbase + blk) + __popcll(m & ((1ull << c) - 1ull));
    return xr >= r0 && xr < r1;
  }
  return owns_row(row, b0, b1);
}

// The vectors only their own CTA touches between true residuals, p and x, stay
// in shared memory for as many of its chunks as fit: the passes of a large solve
// wait for L2 (9 TB/s in FP64, 28 % of its peak), and p is 2 of pass A's 5 streams,
// x 2 of pass E's 8.  On 20,834 blocks this measured FP64 48.5 -> 41.8 us, mixed 38.1 -> 36.5 us
// an iteration.  A chunk of p is a slot of kSlotBytes (16 bytes a lane, the fragment
// layout), a chunk of x CB slots in cell order.  p fills the slots first.
constexpr int kSlotBytes = 512;

template <class T, bool RES>
struct Resident {
  T* p;       // chunk c < np of p
  double* x;  // chunk c < nx of x
  int np, nx;
  bool any;   // whether the launch has slots at all (the same for the team)
  __device__ __forceinline__ Resident(unsigned char* base, int slots, int b0, int b1) {
    const int nch = (b1 - b0 + Frag<T>::CB - 1) / Frag<T>::CB;
    np = RES ? min(nch, slots) : 0;
    nx = RES ? min(nch, (slots - np) / Frag<T>::CB) : 0;
    p = reinterpret_cast<T*>(base);
    x = reinterpret_cast<double*>(base + (size_t)np * kSlotBytes);
    any = RES && slots > 0;
  }
  __device__ __forceinline__ T* p_at(int c, int lane) const { return p + (c * 32 + lane) * Frag<T>::N; }
  // the two functions below copy whole chunks; all threads, then synchronise
  __device__ __forceinline__ void fetch_x(const double* __restrict__ g, int b0, int b1) const {
    const int n = min(nx * Frag<T>::CB, b1 - b0) * kBLEN;
    for (int i = 2 * (int)threadIdx.x; i < n; i += 2 * kSolveThreads)
      *reinterpret_cast<double2*>(x + i) = __ldcg(reinterpret_cast<const double2*>(g + b0 * kBLEN + i));
  }
  __device__ __forceinline__ void put_x(double* __restrict__ g, int b0, int b1) const {
    const int n = min(nx * Frag<T>::CB, b1 - b0) * kBLEN;
    for (int i = 2 * (int)threadIdx.x; i < n; i += 2 * kSolveThreads)
      *reinterpret_cast<double2*>(g + b0 * kBLEN + i) = *reinterpret_cast<const double2*>(x + i);
  }
};

struct IterState {
  double rho, nr, nrh;  // (rhat,r), |r|^2, |rhat|^2 of the current residual
  double err_init;      // L-inf norm the relative test divides by
  double err_opt;       // best residual norm seen (FP64: recursive; mixed: true)
  double err_true;      // mixed: last true residual |b - A x|_inf
  int restarts;
  int iters;
  int updates;          // mixed: true-residual replacements
  int status;
  bool best_is_x;
};

__device__ __forceinline__ double dprod(double a, double b) { return a * b; }
__device__ __forceinline__ double dprod(float a, float b) { return (double)a * (double)b; }

// SpMV epilogue of pass B: nu = y, (rhat, nu).
template <class T>
struct EpiRhNu {
  static constexpr int LV = Lane<T>::V;
  const T* rh;
  T* nu;
  double acc;
  struct Pre {
    T v[LV];  // rhat
  };
  __device__ __forceinline__ Pre load(int i0) const {
    Pre p;
    ldv<LV>(rh + i0, p.v);
    return p;
  }
  __device__ __forceinline__ Pre load1(int i) const {
    Pre p{};
    p.v[0] = __ldcg(rh + i);
    return p;
  }
  __device__ __forceinline__ void vec(int i0, const T (&y)[LV], const Pre& p) {
    stv<LV>(nu + i0, y);
#pragma unroll
    for (int j = 0; j < LV; ++j) acc += dprod(p.v[j], y[j]);
  }
  __device__ __forceinline__ void one(int i, T y, const Pre& p, int j) {
    nu[i] = y;
    acc += dprod(p.v[j], y);
  }
};

// SpMV epilogue of pass D: t = y, (t, s), (t, t).
template <class T>
struct EpiTS {
  static constexpr int LV = Lane<T>::V;
  const T* s;
  T* t;
  double ts, tt;
  struct Pre {
    T v[LV];  // s
  };
  __device__ __forceinline__ Pre load(int i0) const {
    Pre p;
    ldv<LV>(s + i0, p.v);
    return p;
  }
  __device__ __forceinline__ Pre load1(int i) const {
    Pre p{};
    p.v[0] = __ldcg(s + i);
    return p;
  }
  __device__ __forceinline__ void vec(int i0, const T (&y)[LV], const Pre& p) {
    stv<LV>(t + i0, y);
#pragma unroll
    for (int j = 0; j < LV; ++j) {
      ts += dprod(y[j], p.v[j]);
      tt += dprod(y[j], y[j]);
    }
  }
  __device__ __forceinline__ void one(int i, T y, const Pre& p, int j) {
    t[i] = y;
    ts += dprod(y, p.v[j]);
    tt += dprod(y, y);
  }
};

// Mixed form: r = (b - mean_b) - A x in FP64, stored as FP32 (and as rhat
// when set_rh); B.out: |r64|_inf, (rhat,r), |r|^2, |rhat|^2, |r32|_inf over the
// team.  x must be visible to the team.  Returns false if the wait gave up.
template <class SM>
__device__ __forceinline__ bool true_residual(SM& sm, Team& B, const MeshView& M, const double* __restrict__ b,
                                              double mean_b, const double* __restrict__ x, float* __restrict__ r,
                                              float* __restrict__ rh, bool set_rh, int b0, int b1, int r0, int r1,
                                              int phase) {
  struct Epi {
    const double* b;
    double mean_b;
    float* r;
    float* rh;
    bool set_rh;
    double v[5];
    struct Pre {
      double b[2];
      float rh[2];
    };
    __device__ __forceinline__ Pre load(int i0) const {
      Pre p;
      ldv<2>(b + i0, p.b);
      if (set_rh) p.rh[0] = p.rh[1] = 0.f;
      else ldv<2>(rh + i0, p.rh);
      return p;
    }
    __device__ __forceinline__ Pre load1(int i) const {
      Pre p{};
      p.b[0] = __ldg(b + i);
      if (!set_rh) p.rh[0] = __ldcg(rh + i);
      return p;
    }
    __device__ __forceinline__ float acc(double y, double bi, float rhi) {
      const double r64 = (bi - mean_b) - y;
      const float r32 = (float)r64;
      const float rhv = set_rh ? r32 : rhi;
      v[0] = nanmax(v[0], fabs(r64));
      v[1] += dprod(rhv, r32);
      v[2] += dprod(r32, r32);
      v[3] += dprod(rhv, rhv);
      v[4] = nanmax(v[4], fabs((double)r32));
      return r32;
    }
    __device__ __forceinline__ void vec(int i0, const double (&y)[2], const Pre& p) {
      float rr[2];
      rr[0] = acc(y[0], p.b[0], p.rh[0]);
      rr[1] = acc(y[1], p.b[1], p.rh[1]);
      stv<2>(r + i0, rr);
      if (set_rh) stv<2>(rh + i0, rr);
    }
    __device__ __forceinline__ void one(int i, double y, const Pre& p, int j) {
      const float r32 = acc(y, p.b[j], p.rh[j]);
      r[i] = r32;
      if (set_rh) rh[i] = r32;
    }
  } epi{b, mean_b, r, rh, set_rh, {0.0, 0.0, 0.0, 0.0, 0.0}};
  spmv_range<double>(M, x, b0, b1, r0, r1, epi, spmv_row(sm));
  return B.reduce<5>(epi.v, 0x11u, phase);
}

struct MixedCtx {  // what the reliable update needs
  const double* b;
  double mean_b;
  double delta;
  double tol_abs, tol_rel;
  bool restart;  // restart the recurrences at each replacement
};

// Runs BiCGSTABSolver::main's loop from a prepared state (r, rhat = r,
// st.rho/nr/nrh/err_init set, p = nu = 0 implied).  T is the Krylov type,
// X the solution type; RU enables the mixed form's true-residual
// replacement; MC the mean constraint (FP64 only); AHEAD the operands of
// passes A and C one chunk ahead.  Returns false if a barrier gave up.
template <class T, bool RU, bool MC, bool AHEAD, bool RES>
__device__ bool bicgstab_loop(Smem<T>& sm, Team& B, const SineSolve<T>& pin, const Problem<T>& V,
                              const Resident<T, RES>& R, int b0, int b1, int r0, int r1, const SolveParams& sp,
                              const MixedCtx& mx, IterState& st) {
  static_assert(!(MC && RU), "the mean constraint runs in the FP64 form only");
  using X = double;
  const MeshView& M = V.M;
  constexpr int LV = Lane<T>::V, CB = Lane<T>::CB;  // 16-byte lane layout
  constexpr int FN = Frag<T>::N;                    // values per lane in the fragment layout of passes A and C
  static_assert(CB == Frag<T>::CB, "the layouts share the chunk");
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const Lane<T> L(lane);
  T* const scratch = warp_scratch(sm);
  const double eps = 1e-21;
  // MC: the CTA whose SpMV computes the mean row records that row's own
  // product (its partials subtract it and add the sum h^2 v in its place)
  const bool rec_mean = MC && computes_row(M, sp.mean_row, b0, b1, r0, r1);
  double rho_prev = 1.0, alpha = 1.0, omega = 1.0, beta;
  bool zero_pnu = true;
  double rho = st.rho, nr = st.nr, nrh = st.nrh;
  double rmax_since = sqrt(nr);  // largest |r|_2 since the last true residual
  int since = 0;                 // iterations since the last true residual
  int k;
  st.status = CUP2D_NOT_CONVERGED;
  for (k = 0; k < sp.max_iter; ++k) {
    // scalar step (BiCGSTAB.cu:471-509)
    const bool serious_breakdown = rho * rho < 1e-16 * nr * nrh;
    beta = (rho / (rho_prev + eps)) * (alpha / (omega + eps));
    bool restart_now = false;
    if (serious_breakdown && sp.max_restarts > 0) {
      ++st.restarts;
      if (st.restarts >= sp.max_restarts) { st.status = CUP2D_BREAKDOWN_LIMIT; break; }
      restart_now = true;
      rho = nr;  // |rhat|^2 after rhat = r
      nrh = nr;
      zero_pnu = true;
      rho_prev = 1.0; alpha = 1.0; omega = 1.0;
      beta = (rho / (rho_prev + eps)) * (alpha / (omega + eps));
    }
    const T tb_beta = (T)beta, tb_omega = (T)omega;
    // pass A: p = r + beta (p - omega nu); z = P^-1 p, warp by warp.  AHEAD:
    // the next chunk's operands are loaded before this chunk's block solve, so
    // that the loads overlap it.
    {
      T rr[FN], pp[FN], nn[FN];
      auto load = [&](int c) {
        const int blk = b0 + c * CB, nv = b1 - blk;
        ld_frag<T>(V.r, blk, nv, lane, rr);
        if (!zero_pnu) {
          if (RES && c < R.np) lds16<FN>(R.p_at(c, lane), pp);
          else ld_frag<T>(V.p, blk, nv, lane, pp);
          ld_frag<T>(V.nu, blk, nv, lane, nn);
        }
      };
      const int nch = (b1 - b0 + CB - 1) / CB;
      if (AHEAD && w < nch) load(w);
      for (int c = w; c < nch; c += kWarps) {
        if (!AHEAD) load(c);
        const int blk = b0 + c * CB, nv = b1 - blk;
        T pv[FN];
#pragma unroll
        for (int k = 0; k < FN; ++k) pv[k] = zero_pnu ? rr[k] : rr[k] + tb_beta * (pp[k] - tb_omega * nn[k]);
        if (restart_now) st_frag<T>(V.rh, blk, nv, lane, rr);
        if (RES && c < R.np) stv<FN>(R.p_at(c, lane), pv);
        else st_frag<T>(V.p, blk, nv, lane, pv);
        if (AHEAD && c + kWarps < nch) load(c + kWarps);
        pin.apply(pv, scratch, lane);
        st_frag<T>(V.z, blk, nv, lane, pv);
      }
      zero_pnu = false;
    }
    if (!B.sync(1)) return false;
    // pass B: nu = A z; (rhat, nu)
    double rhnu;
    {
      EpiRhNu<T> epi{V.rh, V.nu, 0.0};
      spmv_range_staged<T>(M, V.z, V.rh, b0, b1, r0, r1, epi, spmv_stage(sm));
      if constexpr (MC) {
        // the mean row's own product and rhat, to swap in sum h^2 z below
        double v[4] = {epi.acc, hsum_part(M, V.z, b0, b1), 0.0, 0.0};
        __syncthreads();
        if (threadIdx.x == 0 && rec_mean) {
          const T y = __ldcg(V.nu + sp.mean_row), rv = __ldcg(V.rh + sp.mean_row);
          v[2] = dprod(rv, y);
          v[3] = (double)rv;
        }
        if (!B.reduce<4>(v, 0u, 2)) return false;
        const double* const o = B.out;
        const T m = (T)o[1];
        rhnu = (o[0] - o[2]) + o[3] * (double)m;
        if (threadIdx.x == 0 && owns_row(sp.mean_row, b0, b1)) V.nu[sp.mean_row] = m;
        __syncthreads();
      } else {
        const double v[1] = {epi.acc};
        if (!B.reduce<1>(v, 0u, 2)) return false;
        rhnu = B.out[0];
      }
    }
    alpha = rho / (rhnu + eps);
    const T ta = (T)alpha;
    // pass C: s = r - alpha nu (in place of r); z2 = P^-1 s
    {
      T rr[FN], nn[FN];
      auto load = [&](int blk) {
        ld_frag<T>(V.r, blk, b1 - blk, lane, rr);
        ld_frag<T>(V.nu, blk, b1 - blk, lane, nn);
      };
      int blk = b0 + w * CB;
      if (AHEAD && blk < b1) load(blk);
      for (; blk < b1; blk += kWarps * CB) {
        if (!AHEAD) load(blk);
        const int nv = b1 - blk;
        T sv[FN];
#pragma unroll
        for (int k = 0; k < FN; ++k) sv[k] = rr[k] - ta * nn[k];
        st_frag<T>(V.r, blk, nv, lane, sv);
        if (AHEAD && blk + kWarps * CB < b1) load(blk + kWarps * CB);
        pin.apply(sv, scratch, lane);
        st_frag<T>(V.z2, blk, nv, lane, sv);
      }
    }
    if (!B.sync(3)) return false;
    // pass D: t = A z2; (t,s), (t,t)
    {
      EpiTS<T> epi{V.r, V.t, 0.0, 0.0};
      spmv_range_staged<T>(M, V.z2, V.r, b0, b1, r0, r1, epi, spmv_stage(sm));
      if constexpr (MC) {
        double v[6] = {epi.ts, epi.tt, hsum_part(M, V.z2, b0, b1), 0.0, 0.0, 0.0};
        __syncthreads();
        if (threadIdx.x == 0 && rec_mean) {
          const T y = __ldcg(V.t + sp.mean_row), sv = __ldcg(V.r + sp.mean_row);
          v[3] = dprod(y, sv);
          v[4] = dprod(y, y);
          v[5] = (double)sv;
        }
        if (!B.reduce<6>(v, 0u, 4)) return false;
        const double* const o = B.out;
        const T m = (T)o[2];
        const double ts = (o[0] - o[3]) + o[5] * (double)m;
        const double tt = (o[1] - o[4]) + dprod(m, m);
        omega = ts / (tt + eps);
        if (threadIdx.x == 0 && owns_row(sp.mean_row, b0, b1)) V.t[sp.mean_row] = m;
        __syncthreads();
      } else {
        const double v[2] = {epi.ts, epi.tt};
        if (!B.reduce<2>(v, 0u, 4)) return false;
        omega = B.out[0] / (B.out[1] + eps);
      }
    }
    const T to = (T)omega;
    // pass E: x += alpha z, then x += omega z2 (the reference's two axpys,
    // fused into one pass); r = s - omega t; norms.  The best iterate is
    // saved lazily here: x still holds the previous iterate.  One chunk per
    // warp step: two chunks in flight kept twice the vectors live across the
    // loads, and the spills this forced slowed every pass of the kernel
    // (measured: 12 % on the mixed batch, 20 % on a large FP64 solve).
    {
      double v[4] = {0.0, 0.0, 0.0, 0.0};
      const int nch = (b1 - b0 + CB - 1) / CB;
      for (int c = w; c < nch; c += kWarps) {
        const int blk = b0 + c * CB + L.bl;
        if (blk >= b1) continue;
        const int i0 = blk * kBLEN + L.cell0;
        X xv[LV];
        T zv[LV], z2v[LV], sv[LV], tv[LV], rhv[LV];
        double* const xs = R.x + (c * CB + L.bl) * kBLEN + L.cell0;  // where chunk c of x is resident
        if (RES && c < R.nx) {
#pragma unroll
          for (int k = 0; k < LV; k += 2) {
            const double2 a = *reinterpret_cast<const double2*>(xs + k);
            xv[k] = a.x;
            xv[k + 1] = a.y;
          }
        } else {
          ldv<LV>(V.x + i0, xv);
        }
        ldv<LV>(V.z + i0, zv);
        ldv<LV>(V.z2 + i0, z2v);
        ldv<LV>(V.r + i0, sv);
        ldv<LV>(V.t + i0, tv);
        ldv<LV>(V.rh + i0, rhv);
        if (st.best_is_x) stv<LV>(V.xo + i0, xv);
        X xn[LV];
        T rn[LV];
#pragma unroll
        for (int k = 0; k < LV; ++k) {
          const X x1 = xv[k] + (X)alpha * (X)zv[k];
          xn[k] = x1 + (X)omega * (X)z2v[k];
          rn[k] = sv[k] - to * tv[k];
          v[0] = nanmax(v[0], fabs((double)rn[k]));
          v[1] += dprod(rhv[k], rn[k]);
          v[2] += dprod(rn[k], rn[k]);
          v[3] += dprod(rhv[k], rhv[k]);
        }
        stv<LV>(RES && c < R.nx ? xs : V.x + i0, xn);
        stv<LV>(V.r + i0, rn);
      }
      if (!B.reduce<4>(v, 0x1u, 5)) return false;
    }
    double error = B.out[0];
    double rho_new = B.out[1];
    nr = B.out[2];
    nrh = B.out[3];
    if (!(error == error) || !(rho_new == rho_new)) {  // non-finite: stop, keep the best iterate
      st.best_is_x = false;
      ++k;
      break;
    }
    bool refreshed = false;
    if constexpr (RU) {
      rmax_since = fmax(rmax_since, sqrt(nr));
      ++since;
      const bool claims = (error <= sp.tol_abs) || (error / st.err_init <= sp.tol_rel);
      // refresh when the FP32 residual dropped by delta, claims convergence,
      // or a sweep stalls for kMaxSweep iterations
      if (claims || sqrt(nr) < mx.delta * rmax_since || since >= kMaxSweep) {
        since = 0;
        // pass E's barrier already ordered every CTA's x update before this,
        // but for what is resident
        if (RES && R.any) {
          R.put_x(V.x, b0, b1);
          if (!B.sync(6)) return false;
        }
        if (!true_residual(sm, B, M, mx.b, mx.mean_b, V.x, V.r, V.rh, mx.restart, b0, b1, r0, r1, 6)) return false;
        ++st.updates;
        refreshed = true;
        st.err_true = B.out[0];
        rho_new = B.out[1];
        nr = B.out[2];
        nrh = B.out[3];
        error = B.out[4];
        rmax_since = sqrt(nr);
        if ((st.err_true <= mx.tol_abs) || (st.err_true / st.err_init <= mx.tol_rel)) {
          st.err_opt = fmin(st.err_opt, st.err_true);
          st.best_is_x = true;
          st.status = CUP2D_OK;
          ++k;
          break;
        }
      }
    }
    // convergence (BiCGSTAB.cu:571-600)
    if constexpr (RU) {
      // mixed: an iterate is judged by its true residual, which only a
      // refresh computes (err_opt is the best true residual so far).  x
      // moves in every pass E, so between refreshes the best iterate is the
      // copy in xo, written by the pass E after the refresh that found it:
      // one copy per refresh, not one per iteration
      st.best_is_x = refreshed && st.err_true < st.err_opt;
      if (st.best_is_x) st.err_opt = st.err_true;
    } else if (error < st.err_opt) {
      st.err_opt = error;
      st.best_is_x = true;
      if ((error <= sp.tol_abs) || (error / st.err_init <= sp.tol_rel)) {
        st.status = CUP2D_OK;
        ++k;
        break;
      }
    } else {
      st.best_is_x = false;
    }
    if (RU && refreshed && mx.restart) {
      // rhat = r was written with the true residual: fresh recurrences
      rho_prev = 1.0; alpha = 1.0; omega = 1.0;
      rho = rho_new;
      zero_pnu = true;
    } else {
      rho_prev = rho;
      rho = rho_new;
    }
  }
  st.iters += k;
  return true;
}

// x -= sum(h^2 x)/sum(h^2) over the CTA's blocks (ExpAMRSolver.cpp:383-415);
// x already holds the final iterate.
template <class SM>
__device__ bool subtract_mean(SM& sm, Team& B, const MeshView& M, double* __restrict__ x,
                              int b0, int b1) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double v[2] = {0.0, 0.0};
  for (int blk = b0 + w; blk < b1; blk += kWarps) {
    const int o = blk * kBLEN;
    const double hb = __ldg(M.hblk + blk);
    v[0] += (__ldcg(x + o + lane) + __ldcg(x + o + lane + 32)) * (hb * hb);
    v[1] += 2.0 * (hb * hb);
  }
  if (!B.reduce<2>(v, 0u, 7)) return false;
  const double avg = B.out[0] / B.out[1];
  for (int blk = b0 + w; blk < b1; blk += kWarps) {
    const int o = blk * kBLEN;
    x[o + lane] = __ldcg(x + o + lane) - avg;
    x[o + lane + 32] = __ldcg(x + o + lane + 32) - avg;
  }
  return true;
}

// x <- x_opt when the last iterate was not the best
__device__ __forceinline__ void take_best(bool best_is_x, double* __restrict__ x, const double* __restrict__ xo,
                                          int b0, int b1) {
  if (best_is_x) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int blk = b0 + w; blk < b1; blk += kWarps) {
    const int o = blk * kBLEN;
    x[o + lane] = __ldcg(xo + o + lane);
    x[o + lane + 32] = __ldcg(xo + o + lane + 32);
  }
}

// The kernels' dynamic shared memory: Smem<T>, then the resident slots.
extern __shared__ __align__(16) unsigned char g_solve_smem[];
static_assert(sizeof(Smem<float>) % 16 == 0 && sizeof(Smem<double>) % 16 == 0, "16-byte slots");
template <class T>
__device__ __forceinline__ Smem<T>& solve_smem() {
  return *reinterpret_cast<Smem<T>*>(g_solve_smem);
}

// ============================================ one problem, one team ========

__device__ __forceinline__ void write_stats(const Team& B, DevStats* stats, const IterState& st, int refinements,
                                            double err_final, double norm_ax0) {
  if (B.rank == 0 && threadIdx.x == 0) {
    stats->status = st.status;
    stats->iterations = st.iters;
    stats->restarts = st.restarts;
    stats->refinements = refinements;
    stats->err_init = st.err_init;
    stats->err_opt = err_final;
    stats->norm_ax0 = norm_ax0;
  }
}

// Plain FP64 solve of one problem by the team: BiCGSTABSolver::main
// (BiCGSTAB.cu:412-620) and the mean removal (ExpAMRSolver.cpp:383-415).
// [b0,b1) is this CTA's block range, [r0,r1) its explicit rows.
// MC: the mean constraint (sp.mean_row).
template <bool MC, bool RES, bool AHEAD = true>
__device__ bool solve_fp64(Smem<double>& sm, Team& B, const SineSolve<double>& pin, const Problem64& pr,
                           const SolveParams& sp, int slots, int b0, int b1, int r0, int r1) {
  const MeshView& M = pr.M;
  const Resident<double, RES> R(g_solve_smem + sizeof(Smem<double>), slots, b0, b1);
  if constexpr (RES) R.fetch_x(pr.x, b0, b1);  // read after the first reduction's barriers
  double x0sum = 0.0;  // MC: sum h^2 x0, the mean row of A x0
  if constexpr (MC) {
    const double v[1] = {hsum_part(M, pr.x, b0, b1)};
    if (!B.reduce<1>(v, 0u, 9)) return false;
    x0sum = B.out[0];
  }
  // r = b - A x0, rhat = r, |A x0|_inf, |r0|_inf (BiCGSTAB.cu:430-465)
  {
    struct Epi {
      const double* b;
      double* r;
      double* rh;
      int mrow;
      double msum;
      double v[3];
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
      __device__ __forceinline__ double acc(double y, double bi) {
        const double rv = bi - y;
        v[0] = nanmax(v[0], fabs(y));
        v[1] = nanmax(v[1], fabs(rv));
        v[2] += rv * rv;
        return rv;
      }
      // the mean row: (A x0) reads sum h^2 x0, b reads 0 (getVec, ExpAMRSolver.cpp:340-346)
      __device__ __forceinline__ double accm(int i, double y, double bi) {
        return (MC && i == mrow) ? acc(msum, 0.0) : acc(y, bi);
      }
      __device__ __forceinline__ void vec(int i0, const double (&y)[2], const Pre& p) {
        double rr[2];
        rr[0] = accm(i0, y[0], p.b[0]);
        rr[1] = accm(i0 + 1, y[1], p.b[1]);
        stv<2>(r + i0, rr);
        stv<2>(rh + i0, rr);
      }
      __device__ __forceinline__ void one(int i, double y, const Pre& p, int j) {
        const double rv = accm(i, y, p.b[j]);
        r[i] = rv;
        rh[i] = rv;
      }
    } epi{pr.b, pr.r, pr.rh, sp.mean_row, x0sum, {0.0, 0.0, 0.0}};
    spmv_range<double>(M, pr.x, b0, b1, r0, r1, epi, spmv_row(sm));
    if (!B.reduce<3>(epi.v, 0x3u, 0)) return false;
  }
  IterState st;
  const double norm_ax0 = B.out[0];
  st.err_init = B.out[1];
  st.err_opt = st.err_init;
  st.err_true = st.err_init;
  st.rho = st.nr = st.nrh = B.out[2];
  st.restarts = 0;
  st.iters = 0;
  st.updates = 0;
  st.best_is_x = true;
  st.status = CUP2D_NOT_CONVERGED;
  const MixedCtx none{};
  if (!bicgstab_loop<double, false, MC, AHEAD, RES>(sm, B, pin, pr, R, b0, b1, r0, r1, sp, none, st))
    return false;
  if (RES && R.any && st.best_is_x) {
    R.put_x(pr.x, b0, b1);
    __syncthreads();
  }
  take_best(st.best_is_x, pr.x, pr.xo, b0, b1);
  if (sp.subtract_mean && !subtract_mean(sm, B, M, pr.x, b0, b1)) return false;
  write_stats(B, pr.stats, st, 0, st.err_opt, norm_ax0);
  return true;
}

// Mixed-precision solve of one problem by the team.
template <bool RES>
__device__ bool solve_mixed(Smem<float>& sm, Team& B, const SineSolve<float>& pin, const ProblemMixed& pr,
                            const SolveParams& sp, int slots, int b0, int b1, int r0, int r1) {
  const Resident<float, RES> R(g_solve_smem + sizeof(Smem<float>), slots, b0, b1);
  if constexpr (RES) R.fetch_x(pr.x, b0, b1);  // read after the first reduction's barriers
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // Neumann compatibility: project b to zero sum (sum b / n)
  {
    double v[1] = {0.0};
    for (int blk = b0 + w; blk < b1; blk += kWarps) {
      const int o = blk * kBLEN;
      v[0] += __ldg(pr.b + o + lane) + __ldg(pr.b + o + lane + 32);
    }
    if (!B.reduce<1>(v, 0u, 8)) return false;
  }
  MixedCtx mx;
  mx.b = pr.b;
  mx.mean_b = B.out[0] / (double)(pr.M.nb * kBLEN);
  mx.delta = sp.reliable_delta;
  mx.tol_abs = sp.tol_abs;
  mx.tol_rel = sp.tol_rel;
  mx.restart = sp.reliable_restart != 0;
  if (!true_residual(sm, B, pr.M, pr.b, mx.mean_b, pr.x, pr.r, pr.rh, true, b0, b1, r0, r1, 0)) return false;
  IterState st;
  st.err_init = B.out[0];
  st.err_true = B.out[0];
  st.err_opt = B.out[0];  // best true residual: x0's
  st.rho = B.out[1];
  st.nr = B.out[2];
  st.nrh = B.out[3];
  st.restarts = 0;
  st.iters = 0;
  st.updates = 0;
  st.best_is_x = true;
  st.status = CUP2D_NOT_CONVERGED;
  const bool done0 = st.err_true <= sp.tol_abs || st.err_true == 0.0;
  if (done0) {
    st.status = CUP2D_OK;
  } else if (!bicgstab_loop<float, true, false, true, RES>(sm, B, pin, pr, R, b0, b1, r0, r1, sp, mx, st)) {
    return false;
  }
  take_best(st.best_is_x, pr.x, pr.xo, b0, b1);
  if (sp.subtract_mean && !subtract_mean(sm, B, pr.M, pr.x, b0, b1)) return false;
  write_stats(B, pr.stats, st, st.updates, st.status == CUP2D_OK ? st.err_true : st.err_opt, 0.0);
  return true;
}

}  // namespace

// ====================================================== single solves =====

// kSolveCtasPerSm CTAs per SM (2: up to 128 registers, no spills).  With the
// SpMV operands staged in shared memory the spill-free build gained 6-7 % per
// iteration on the large workload and ~10 % on time stepping over 3 CTAs at
// 80 registers (an earlier kernel, gathering its operands into registers,
// had measured 97/95/104 us per iteration at 2/3/4).
__global__ void __launch_bounds__(kSolveThreads, kSolveCtasPerSm) k_bicgstab64(const __grid_constant__ SolveArgs64 S) {
  Smem<double>& sm = solve_smem<double>();
  const int b0 = share(S.prob.M.nb, blockIdx.x, gridDim.x), b1 = share(S.prob.M.nb, blockIdx.x + 1, gridDim.x);
  const int r0 = share(S.prob.M.R, blockIdx.x, gridDim.x), r1 = share(S.prob.M.R, blockIdx.x + 1, gridDim.x);
  Team& B = sm.team;
  if (threadIdx.x == 0) B.init(blockIdx.x, gridDim.x, S.bar, S.red, S.abort_flag, S.timeout_ns, S.prof);
  SineSolve<double> pin;
  pin.init();
  __syncthreads();
  solve_fp64<false, true>(sm, B, pin, S.prob, S.sp, S.nslots, b0, b1, r0, r1);
}

// With bMeanConstraint: the same solve on the system whose row S.sp.mean_row
// is sum h^2 x = 0.
__global__ void __launch_bounds__(kSolveThreads, kSolveCtasPerSm)
    k_bicgstab64_mean(const __grid_constant__ SolveArgs64 S) {
  Smem<double>& sm = solve_smem<double>();
  const int b0 = share(S.prob.M.nb, blockIdx.x, gridDim.x), b1 = share(S.prob.M.nb, blockIdx.x + 1, gridDim.x);
  const int r0 = share(S.prob.M.R, blockIdx.x, gridDim.x), r1 = share(S.prob.M.R, blockIdx.x + 1, gridDim.x);
  Team& B = sm.team;
  if (threadIdx.x == 0) B.init(blockIdx.x, gridDim.x, S.bar, S.red, S.abort_flag, S.timeout_ns, S.prof);
  SineSolve<double> pin;
  pin.init();
  __syncthreads();
  solve_fp64<true, true>(sm, B, pin, S.prob, S.sp, S.nslots, b0, b1, r0, r1);
}

__global__ void __launch_bounds__(kSolveThreads, kSolveCtasPerSm) k_bicgstab_mixed(const __grid_constant__ SolveArgsMixed S) {
  Smem<float>& sm = solve_smem<float>();
  const int b0 = share(S.prob.M.nb, blockIdx.x, gridDim.x), b1 = share(S.prob.M.nb, blockIdx.x + 1, gridDim.x);
  const int r0 = share(S.prob.M.R, blockIdx.x, gridDim.x), r1 = share(S.prob.M.R, blockIdx.x + 1, gridDim.x);
  Team& B = sm.team;
  if (threadIdx.x == 0) B.init(blockIdx.x, gridDim.x, S.bar, S.red, S.abort_flag, S.timeout_ns, S.prof);
  SineSolve<float> pin;
  pin.init();
  __syncthreads();
  solve_mixed<true>(sm, B, pin, S.prob, S.sp, S.nslots, b0, b1, r0, r1);
}


// The server's instances of the two single solves: the same bodies at
// kServedCtasPerSm CTAs per SM.
__global__ void __launch_bounds__(kSolveThreads, kServedCtasPerSm)
    k_bicgstab64_served(const __grid_constant__ SolveArgs64 S) {
  Smem<double>& sm = solve_smem<double>();
  const int b0 = share(S.prob.M.nb, blockIdx.x, gridDim.x), b1 = share(S.prob.M.nb, blockIdx.x + 1, gridDim.x);
  const int r0 = share(S.prob.M.R, blockIdx.x, gridDim.x), r1 = share(S.prob.M.R, blockIdx.x + 1, gridDim.x);
  Team& B = sm.team;
  if (threadIdx.x == 0) B.init(blockIdx.x, gridDim.x, S.bar, S.red, S.abort_flag, S.timeout_ns, S.prof);
  SineSolve<double> pin;
  pin.init();
  __syncthreads();
  solve_fp64<false, false>(sm, B, pin, S.prob, S.sp, 0, b0, b1, r0, r1);
}

__global__ void __launch_bounds__(kSolveThreads, kServedCtasPerSm)
    k_bicgstab_mixed_served(const __grid_constant__ SolveArgsMixed S) {
  Smem<float>& sm = solve_smem<float>();
  const int b0 = share(S.prob.M.nb, blockIdx.x, gridDim.x), b1 = share(S.prob.M.nb, blockIdx.x + 1, gridDim.x);
  const int r0 = share(S.prob.M.R, blockIdx.x, gridDim.x), r1 = share(S.prob.M.R, blockIdx.x + 1, gridDim.x);
  Team& B = sm.team;
  if (threadIdx.x == 0) B.init(blockIdx.x, gridDim.x, S.bar, S.red, S.abort_flag, S.timeout_ns, S.prof);
  SineSolve<float> pin;
  pin.init();
  __syncthreads();
  solve_mixed<false>(sm, B, pin, S.prob, S.sp, 0, b0, b1, r0, r1);
}

// ========================================================= batches ========
//
// Many independent problems in one cooperative launch.  The grid is split
// into groups of `team` consecutive CTAs; each group takes problems from a
// shared queue (largest first, so the tail is short) and solves each one
// with the same code as a single solve, synchronising on its own bounded
// barrier.  All groups share the abort flag: a timeout anywhere ends the
// launch.

template <bool MIXED>
__device__ __forceinline__ void batch_body(const BatchArgs& A) {
  using KT = typename std::conditional<MIXED, float, double>::type;
  Smem<KT>& sm = solve_smem<KT>();
  const int team = A.team;
  const int g = blockIdx.x / team, rank = blockIdx.x % team;
  Team& B = sm.team;
  if (threadIdx.x == 0)
    B.init((unsigned)rank, (unsigned)team, A.bars + g, A.red + (size_t)g * kRedWords * team, A.abort_flag, A.timeout_ns,
           A.prof);
  SineSolve<KT> pin;
  pin.init();
  __syncthreads();
  while (true) {
    if (rank == 0 && threadIdx.x == 0) A.slots[g] = atomicAdd(A.queue, 1);
    if (!B.sync(9)) return;
    unsigned long long t_begin = 0;
    if (threadIdx.x == 0) {
      t_begin = globaltimer_ns();
      sm.slot = __ldcg(A.slots + g);
    }
    __syncthreads();
    const int q = sm.slot;
    if (q >= A.nprob) return;
    const int p = __ldg(A.order + q);
    bool ok;
    if constexpr (MIXED) {
      const ProblemMixed& pr = A.pmx[p];
      const int b0 = share(pr.M.nb, rank, team), b1 = share(pr.M.nb, rank + 1, team);
      const int r0 = share(pr.M.R, rank, team), r1 = share(pr.M.R, rank + 1, team);
      ok = solve_mixed<false>(sm, B, pin, pr, A.sp, 0, b0, b1, r0, r1);
    } else {
      const Problem64& pr = A.p64[p];
      const int b0 = share(pr.M.nb, rank, team), b1 = share(pr.M.nb, rank + 1, team);
      const int r0 = share(pr.M.R, rank, team), r1 = share(pr.M.R, rank + 1, team);
      // at 80 registers the operands held ahead are spilled: 23.3 -> 22.3 ms
      // for 40 iterations of 200 problems on teams of 8 without them
      ok = solve_fp64<false, false, false>(sm, B, pin, pr, A.sp, 0, b0, b1, r0, r1);
    }
    if (!ok) return;
    if (rank == 0 && threadIdx.x == 0) {
      DevStats* ds = MIXED ? A.pmx[p].stats : A.p64[p].stats;
      ds->t_begin = t_begin;
      ds->t_end = globaltimer_ns();
    }
  }
}

__global__ void __launch_bounds__(kSolveThreads, kBatch64CtasPerSm) k_bicgstab_batch64(const __grid_constant__ BatchArgs A) {
  batch_body<false>(A);
}

__global__ void __launch_bounds__(kSolveThreads, kBatchMixedCtasPerSm) k_bicgstab_batch_mixed(const __grid_constant__ BatchArgs A) {
  batch_body<true>(A);
}

// ------------------------------------------------------------ launch -----

namespace {
constexpr int kNumSolveFns = 7;
const void* const kSolveFns[kNumSolveFns] = {(const void*)k_bicgstab64,        (const void*)k_bicgstab_mixed,
                                             (const void*)k_bicgstab_batch64,  (const void*)k_bicgstab_batch_mixed,
                                             (const void*)k_bicgstab64_mean,   (const void*)k_bicgstab64_served,
                                             (const void*)k_bicgstab_mixed_served};
// CTAs per SM each kernel is built for
const int kSolveFnCtas[kNumSolveFns] = {kSolveCtasPerSm,  kSolveCtasPerSm,  kBatch64CtasPerSm, kBatchMixedCtasPerSm,
                                        kSolveCtasPerSm,  kServedCtasPerSm, kServedCtasPerSm};

int fn_index(const void* fn) {
  int k = 0;
  while (k < kNumSolveFns && kSolveFns[k] != fn) ++k;
  return k;
}

// The kernels with resident slots.
bool resident(const void* fn) {
  return fn == (const void*)k_bicgstab64 || fn == (const void*)k_bicgstab64_mean || fn == (const void*)k_bicgstab_mixed;
}

// Shared memory of a solve kernel beside its resident slots.
size_t base_smem(const void* fn) {
  return (fn == kSolveFns[1] || fn == kSolveFns[3] || fn == kSolveFns[6]) ? sizeof(Smem<float>)
                                                                           : sizeof(Smem<double>);
}

// What a solve kernel may use on a device, queried once per device and kernel
// (handles are created often, e.g. by a server): the largest co-resident grid
// and the resident slots of a CTA.  The plain single solves fill their share of
// the SM's shared memory with slots.  The batches and the served forms have none:
// their vectors stream from HBM and the tables live off L1, which the slots
// would take (512 problems, mixed: 597 ms without, 634 ms with them).
struct FnLimits {
  int grid = 0, slots = 0;
};

cudaError_t query_limits(const void* fn, int dev, FnLimits& out) {
  int per_sm = 0, reserved = 0, optin = 0, sms = 0, ctas = 0;
  cudaError_t e;
  if ((e = cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) != cudaSuccess ||
      (e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess ||
      (e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev)) != cudaSuccess ||
      (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
    return e;
  const int want = kSolveFnCtas[fn_index(fn)];
  const size_t base = base_smem(fn);
  const size_t most = std::min<size_t>(optin, (size_t)per_sm / want - (size_t)reserved);
  const int slots = resident(fn) && most > base ? (int)((most - base) / kSlotBytes) : 0;
  const size_t bytes = base + (size_t)slots * kSlotBytes;
  const int pct = (int)std::min<size_t>(100, (want * (bytes + (size_t)reserved) * 100 + per_sm - 1) / (size_t)per_sm);
  if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes)) != cudaSuccess ||
      (e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, pct)) != cudaSuccess ||
      (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, fn, kSolveThreads, bytes)) != cudaSuccess)
    return e;
  out.grid = sms * ctas;
  out.slots = slots;
  return cudaSuccess;
}

FnLimits fn_limits(const void* fn, int device) {
  static std::atomic<uint64_t> cache[64][kNumSolveFns];
  const int k = fn_index(fn);
  const bool keep = device >= 0 && device < 64;
  if (keep) {
    const uint64_t v = cache[device][k].load(std::memory_order_acquire);
    if (v) return FnLimits{(int)(v >> 32), (int)(uint32_t)v};
  }
  FnLimits l;
  int cur = 0;
  if (cudaGetDevice(&cur) != cudaSuccess) return FnLimits{};
  if (cur != device && cudaSetDevice(device) != cudaSuccess) return FnLimits{};
  const bool ok = query_limits(fn, device, l) == cudaSuccess;
  if (cur != device) cudaSetDevice(cur);
  if (!ok) return FnLimits{};
  if (keep && l.grid > 0)
    cache[device][k].store(((uint64_t)l.grid << 32) | (uint32_t)l.slots, std::memory_order_release);
  return l;
}

// The kernel's limits on the current device; its attributes are set.
cudaError_t current_limits(const void* fn, FnLimits& l) {
  int dev = 0;
  if (cudaError_t e = cudaGetDevice(&dev)) return e;
  l = fn_limits(fn, dev);
  return l.grid > 0 ? cudaSuccess : cudaErrorInvalidConfiguration;
}

// Slots a solve of nb blocks by `grid` CTAs can use: p and x of the largest
// share.
template <class T>
int used_slots(int64_t nb, int grid, int slots) {
  const int64_t nch = ((nb + grid - 1) / grid + Frag<T>::CB - 1) / Frag<T>::CB;
  return (int)std::min<int64_t>(slots, nch * (1 + Frag<T>::CB));
}

int coop_grid(const void* fn, int device) { return fn_limits(fn, device).grid; }
}  // namespace

int max_coop_grid_fp64(int device, bool served) {
  return coop_grid(served ? (const void*)k_bicgstab64_served : (const void*)k_bicgstab64, device);
}
int max_coop_grid_mixed(int device, bool served) {
  return coop_grid(served ? (const void*)k_bicgstab_mixed_served : (const void*)k_bicgstab_mixed, device);
}

int max_coop_grid_mean(int device) { return coop_grid((const void*)k_bicgstab64_mean, device); }

cudaError_t launch_bicgstab64(SolveArgs64& a, int grid, cudaStream_t s, bool served) {
  void* args[] = {&a};
  const void* fn = a.sp.mean_row >= 0 ? (const void*)k_bicgstab64_mean
                   : served           ? (const void*)k_bicgstab64_served
                                      : (const void*)k_bicgstab64;
  FnLimits l;
  if (cudaError_t e = current_limits(fn, l)) return e;
  a.nslots = used_slots<double>(a.prob.M.nb, grid, l.slots);
  return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kSolveThreads), args,
                                     sizeof(Smem<double>) + (size_t)a.nslots * kSlotBytes, s);
}

cudaError_t launch_bicgstab_mixed(SolveArgsMixed& a, int grid, cudaStream_t s, bool served) {
  void* args[] = {&a};
  if (a.sp.mean_row >= 0) return cudaErrorInvalidValue;  // FP64 only
  const void* fn = served ? (const void*)k_bicgstab_mixed_served : (const void*)k_bicgstab_mixed;
  FnLimits l;
  if (cudaError_t e = current_limits(fn, l)) return e;
  a.nslots = used_slots<float>(a.prob.M.nb, grid, l.slots);
  return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kSolveThreads), args,
                                     sizeof(Smem<float>) + (size_t)a.nslots * kSlotBytes, s);
}

int max_coop_grid_batch(int device, bool mixed) {
  return coop_grid(mixed ? (const void*)k_bicgstab_batch_mixed : (const void*)k_bicgstab_batch64, device);
}

// Cooperative launch through the extensible launch API, so that a stream
// capture records the cooperative attribute in the graph's kernel node.
cudaError_t launch_bicgstab_batch(const BatchArgs& a, int grid, bool mixed, cudaStream_t s) {
  void* args[] = {const_cast<BatchArgs*>(&a)};
  const void* fn = mixed ? (const void*)k_bicgstab_batch_mixed : (const void*)k_bicgstab_batch64;
  FnLimits l;
  if (cudaError_t e = current_limits(fn, l)) return e;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kSolveThreads);
  cfg.dynamicSmemBytes = base_smem(fn);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelExC(&cfg, fn, args);
}

// ------------------------------------------------------- single ops -------

// z = P^-1 p, the solve kernels' block solve alone, a warp a chunk.  p and z
// need only their type's alignment.
template <class T>
__device__ __forceinline__ void precond_body(int nb, const T* p, T* z) {
  constexpr int CB = Frag<T>::CB, N = Frag<T>::N;
  __shared__ __align__(16) double scratch[kWarps][kBLEN];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nch = (nb + CB - 1) / CB;
  SineSolve<T> pin;
  pin.init();
  for (int c = (int)blockIdx.x * kWarps + w; c < nch; c += (int)gridDim.x * kWarps) {
    const int i0 = c * CB * kBLEN + Frag<T>::cell0(lane), nv = nb - c * CB;
    T v[N];
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = j / 2 < nv ? p[i0 + (j / 2) * kBLEN + j % 2] : T(0);
    pin.apply(v, reinterpret_cast<T*>(scratch[w]), lane);
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (j / 2 < nv) z[i0 + (j / 2) * kBLEN + j % 2] = v[j];
  }
}

__global__ void __launch_bounds__(kSolveThreads) k_precond64(int nb, const double* p, double* z) {
  precond_body<double>(nb, p, z);
}
__global__ void __launch_bounds__(kSolveThreads) k_precond32(int nb, const float* p, float* z) {
  precond_body<float>(nb, p, z);
}

namespace {
// CTAs for the chunks of nb blocks: enough to fill the device several times.
template <class T>
unsigned precond_grid(int64_t nb) {
  constexpr int64_t per = kWarps * Frag<T>::CB;
  return (unsigned)std::min<int64_t>((nb + per - 1) / per, 4096);
}
}  // namespace

cudaError_t launch_precond64(int64_t nb, const double* p, double* z, cudaStream_t s) {
  if (nb <= 0) return cudaSuccess;
  k_precond64<<<precond_grid<double>(nb), kSolveThreads, 0, s>>>((int)nb, p, z);
  return cudaGetLastError();
}

cudaError_t launch_precond32(int64_t nb, const float* p, float* z, cudaStream_t s) {
  if (nb <= 0) return cudaSuccess;
  k_precond32<<<precond_grid<float>(nb), kSolveThreads, 0, s>>>((int)nb, p, z);
  return cudaGetLastError();
}

}  // namespace cup2d
