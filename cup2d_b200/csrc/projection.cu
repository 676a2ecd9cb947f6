// The pressure projection around the Poisson solve, on the device.
//
// CUP2D's PressureSingle (source/Operators/PressureSingle.cpp) runs three
// field kernels on Cubism block labs (the block plus one ghost layer), each
// followed by Cubism's flux correction on coarse/fine faces:
//   updatePressureRHS  (:324-397)  TMP = facDiv ((u_E - u_W) + (v_N - v_S))
//                                       + (-facDiv CHI) ((ud_E - ud_W) + (vd_N - vd_S)),
//                                  facDiv = 0.5 h / dt
//   updatePressureRHS1 (:399-456)  TMP -= ((p_W + p_E) + (p_S + p_N)) - 4 p
//   pressureCorrection (:123-210)  tmpV = pFac (P_E - P_W, P_N - P_S),
//                                  pFac = -0.5 dt h; V += tmpV (1/h)/h
// Here one warp owns a block, a lane two cells, and evaluates each cell's formula
// in the same order, reading its ghosts straight from the neighbouring blocks:
//   * same-level neighbour: the touching cell;
//   * non-periodic domain edge: velocities flip the sign of the normal
//     component (BlockLabDirichlet, source/Definitions.h:71-196, wall and
//     free-space alike), scalars copy the edge cell (BlockLabNeumann,
//     :200-228);
//   * coarser neighbour: the quadratic interpolation ExpAMRSolver uses for
//     the same cells when it assembles the operator (ExpAMRSolver.cpp:100-128
//     with D1/D2 of ExpAMRSolver.h:268-300), evaluated on values:
//     2/3 close - 1/5 far + 8/15 ((c + sT D1) + D2);
//   * finer neighbours: the mean of the four fine cells the ghost covers.
// The flux correction is folded into the coarse cell's own lane: after its
// formula it adds its own face value (the kernel's storedFace expression with
// that ghost) plus the two fine cells' face values (the same expression from
// the fine side, with their interpolated ghosts).  Cubism, which owns the labs
// and the correction, is an un-vendored submodule of CUP2D; the rules above
// are its role restated from CUP2D's use of it.
//
// The file is compiled without FMA contraction so that every expression
// rounds like the plain IEEE evaluation of the CPU restatement.
//
// Memory: streaming, one pass; per cell the RHS reads vel, udef (16 B each),
// chi, pres (8 B each) and writes tmp, pold (8 B each); the correction reads
// pres (8 B) and updates vel (16 B + 16 B).  Neighbour reads hit L1/L2.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "kernels.hpp"
#include "spmv.cuh"

namespace cup2d {

namespace {

constexpr int kProjThreads = 256;  // 8 warps, a block of 64 cells each at a time
constexpr int kProjWarps = kProjThreads / 32;
constexpr double kI23 = 2. / 3., kI15 = 1. / 5., kI815 = 8. / 15.;

enum : int { kSame = 0, kEdge = 1, kCoarser = 2, kFiner = 3 };

__device__ __forceinline__ int64_t cidx(int64_t blk, int ix, int iy) { return blk * kBLEN + iy * kBS + ix; }

// Cell of block nb across face f (0 W, 1 E, 2 S, 3 N), `d` cells deep, at the
// along-face position of (ix, iy).
__device__ __forceinline__ int64_t mirror(int f, int64_t nb, int ix, int iy, int d) {
  switch (f) {
    case 0: return cidx(nb, kBS - 1 - d, iy);
    case 1: return cidx(nb, d, iy);
    case 2: return cidx(nb, ix, kBS - 1 - d);
    default: return cidx(nb, ix, d);
  }
}

struct Side {
  int kind;
  int64_t blk;      // same-level or coarser block
  int64_t fine[2];  // finer blocks touching cells 0-3 / 4-7 of the face
};

struct Geo {
  ForestView F;
  const int32_t* __restrict__ nbr;

  __device__ int32_t leaf(int l, int64_t i, int64_t j) const {
    if (l < 0 || l >= F.L) return -1;
    return F.table[F.off[l] + j * ((int64_t)F.bpdx << l) + i];
  }

  // The side of face f of block b from the face's neighbour table entry
  // (nbr[4 b + f], loaded ahead by the caller).
  __device__ Side side_from_code(int64_t b, int f, int32_t code) const {
    Side s{kEdge, -1, {-1, -1}};
    if (code >= 0) {
      s.kind = kSame;
      s.blk = code;
      return s;
    }
    if (code != kExplicit) return s;  // domain edge
    const int l = F.level[b];
    const int64_t nx = (int64_t)F.bpdx << l, ny = (int64_t)F.bpdy << l;
    int64_t ni = (int64_t)F.bx[b] + (f == 0 ? -1 : f == 1 ? 1 : 0);
    int64_t nj = (int64_t)F.by[b] + (f == 2 ? -1 : f == 3 ? 1 : 0);
    ni = ni < 0 ? ni + nx : ni >= nx ? ni - nx : ni;  // periodic wrap (one step at most)
    nj = nj < 0 ? nj + ny : nj >= ny ? nj - ny : nj;
    const int32_t c = leaf(l - 1, ni >> 1, nj >> 1);
    if (c >= 0) {
      s.kind = kCoarser;
      s.blk = c;
      return s;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      int64_t ci, cj;
      switch (f) {
        case 0: ci = 2 * ni + 1; cj = 2 * nj + h; break;
        case 1: ci = 2 * ni; cj = 2 * nj + h; break;
        case 2: ci = 2 * ni + h; cj = 2 * nj + 1; break;
        default: ci = 2 * ni + h; cj = 2 * nj; break;
      }
      s.fine[h] = leaf(l + 1, ci, cj);
    }
    // assembly rejected forests with holes; keep every index valid anyway
    s.kind = (s.fine[0] >= 0 && s.fine[1] >= 0) ? kFiner : kEdge;
    return s;
  }
};

// Component c of a field with nc doubles per cell; vector: the component normal
// to the face, whose sign a domain edge flips.
struct Fld {
  const double* __restrict__ p;
  int nc, c;
  bool vector;
  __device__ __forceinline__ double v(int64_t cell) const { return p[cell * nc + c]; }
};

// Ghosts of fine cells from the coarse cell (xc, yc) of block bc:
// ExpAMRSolver::interpolate on values.  The derivatives along the face are
// those of the coarse cell; sT is the fine cell's side of its middle.
struct Interp {
  int64_t c0, c1, c2;
  double a0, a1, a2, b0, b1, b2;
  __device__ __forceinline__ Interp(int64_t bc, int xc, int yc, bool xface) {
    const int t = xface ? yc : xc;
    auto at = [&](int d) { return xface ? cidx(bc, xc, yc + d) : cidx(bc, xc + d, yc); };
    const bool high = t == kBS - 1 || t == kBS / 2 - 1, low = t == 0 || t == kBS / 2;
    c2 = at(0);
    c0 = at(high ? -2 : low ? 2 : -1);
    c1 = at(high ? -1 : 1);
    a0 = high ? 1. / 8. : -1. / 8.;
    a1 = high ? -1. / 2. : low ? 1. / 2. : 1. / 8.;
    a2 = high ? 3. / 8. : low ? -3. / 8. : 0.;
    b0 = 1. / 32.;
    b1 = high || low ? -1. / 16. : 1. / 32.;
    b2 = high || low ? 1. / 32. : -1. / 16.;
  }
  __device__ __forceinline__ double ghost(double v0, double v1, double v2, double vclose, double vfar, double sT) const {
    const double d1 = (a0 * v0 + a1 * v1) + a2 * v2;
    const double d2 = (b0 * v0 + b1 * v1) + b2 * v2;
    const double tay = (v2 + sT * d1) + d2;
    return (kI23 * vclose - kI15 * vfar) + kI815 * tay;
  }
};

// What a face cell needs of one field: its ghost (the lab value), and on a finer
// face for the flux correction its own value, the two fine cells' and the ghosts
// they see.
struct FaceVals {
  double g, own, fine[2], fine_ghost[2];
};

// The ghost cell of one edge cell of block b across face f: ghost gi of the
// block (face gi / 8, cell gi % 8 along it).
struct Ghost {
  const Geo& G;
  int64_t b, cell;
  int ix, iy, f;
  Side s;

  // sd: the face's side, looked up by the caller ahead of its other loads
  __device__ Ghost(const Geo& g, int64_t blk, int gi, const Side& sd) : G(g), b(blk), f(gi >> 3), s(sd) {
    const int k = gi & 7;
    ix = f == 0 ? 0 : f == 1 ? kBS - 1 : k;
    iy = f == 2 ? 0 : f == 3 ? kBS - 1 : k;
    cell = cidx(b, ix, iy);
  }
  __device__ bool xface() const { return f < 2; }
  // fine block and the along-face position of the fine cells facing this cell
  __device__ void fine_cells(int64_t& fb, int& k0) const {
    fb = (xface() ? iy : ix) >= kBS / 2 ? s.fine[1] : s.fine[0];
    k0 = ((xface() ? iy : ix) % (kBS / 2)) * 2;
  }
  // fine cell q (depth d), as a global cell index
  __device__ int64_t fine_cell(int64_t fb, int k0, int q, int d) const {
    return xface() ? mirror(f, fb, 0, k0 + q, d) : mirror(f, fb, k0 + q, 0, d);
  }
  // The values of NF fields, all their loads ahead of the arithmetic.  One by one
  // (a call per field, and per fine cell of a finer face) a warp of a block with
  // coarse/fine faces waited for nine round trips in a row: us for the whole
  // right-hand side 15.3 -> 6.6 on 128 blocks, 28.8 -> 12.7 on 6,000, correction 6.5 -> 3.6
  // and 11.7 -> 5.9.
  template <int NF>
  __device__ __forceinline__ void values(const Fld (&w)[NF], FaceVals (&o)[NF]) const {
    if (s.kind == kSame) {
      const int64_t c = mirror(f, s.blk, ix, iy, 0);
#pragma unroll
      for (int k = 0; k < NF; ++k) o[k].g = w[k].v(c);
    } else if (s.kind == kEdge) {
#pragma unroll
      for (int k = 0; k < NF; ++k) {
        const double own = w[k].v(cell);
        o[k].g = w[k].vector ? -own : own;
      }
    } else if (s.kind == kCoarser) {
      const int64_t bx = G.F.bx[b], by = G.F.by[b];
      const int xc = f == 0 ? kBS - 1 : f == 1 ? 0 : (bx % 2 == 0 ? ix / 2 : ix / 2 + kBS / 2);
      const int yc = f == 2 ? kBS - 1 : f == 3 ? 0 : (by % 2 == 0 ? iy / 2 : iy / 2 + kBS / 2);
      const double sT = xface() ? (iy % 2 == 0 ? -1. : 1.) : (ix % 2 == 0 ? -1. : 1.);
      const int64_t inward = cidx(b, ix + (f == 0 ? 1 : f == 1 ? -1 : 0), iy + (f == 2 ? 1 : f == 3 ? -1 : 0));
      const Interp I(s.blk, xc, yc, xface());
      double v[NF][5];
#pragma unroll
      for (int k = 0; k < NF; ++k) {
        v[k][0] = w[k].v(I.c0);
        v[k][1] = w[k].v(I.c1);
        v[k][2] = w[k].v(I.c2);
        v[k][3] = w[k].v(cell);
        v[k][4] = w[k].v(inward);
      }
#pragma unroll
      for (int k = 0; k < NF; ++k) o[k].g = I.ghost(v[k][0], v[k][1], v[k][2], v[k][3], v[k][4], sT);
    } else {
      int64_t fb;
      int k0;
      fine_cells(fb, k0);
      const int64_t f00 = fine_cell(fb, k0, 0, 0), f01 = fine_cell(fb, k0, 1, 0);
      const int64_t f10 = fine_cell(fb, k0, 0, 1), f11 = fine_cell(fb, k0, 1, 1);
      // seen from the fine block, the interpolation is centred on this cell
      const Interp I(b, ix, iy, xface());
      double v[NF][7];
#pragma unroll
      for (int k = 0; k < NF; ++k) {
        v[k][0] = w[k].v(f00);
        v[k][1] = w[k].v(f01);
        v[k][2] = w[k].v(f10);
        v[k][3] = w[k].v(f11);
        v[k][4] = w[k].v(I.c0);
        v[k][5] = w[k].v(I.c1);
        v[k][6] = w[k].v(I.c2);
      }
#pragma unroll
      for (int k = 0; k < NF; ++k) {
        o[k].g = 0.25 * ((v[k][0] + v[k][1]) + (v[k][2] + v[k][3]));
        o[k].own = v[k][6];
        o[k].fine[0] = v[k][0];
        o[k].fine[1] = v[k][1];
        o[k].fine_ghost[0] = I.ghost(v[k][4], v[k][5], v[k][6], v[k][0], v[k][2], -1.);
        o[k].fine_ghost[1] = I.ghost(v[k][4], v[k][5], v[k][6], v[k][1], v[k][3], 1.);
      }
    }
  }
};

__device__ __forceinline__ double cell_h(const ForestView& F, int l) { return F.h0 / (double)(1ll << l); }

// updatePressureRHS stored face value (PressureSingle.cpp:357-396) of face f
// of a cell: ghost (g, gd), own (w, wd), facDiv and CHI of that cell.
__device__ __forceinline__ double div_face(int f, double facDiv, double chi, double g, double w, double gd, double wd) {
  double s;
  if ((f & 1) == 0) {
    s = facDiv * (g + w);
    s += -(facDiv * chi) * (gd + wd);
  } else {
    s = -facDiv * (g + w);
    s -= -(facDiv * chi) * (gd + wd);
  }
  return s;
}

// pressureCorrectionKernel stored face value (PressureSingle.cpp:152-185).
__device__ __forceinline__ double grad_face(int f, double pFac, double g, double w) {
  return ((f & 1) == 0 ? pFac : -pFac) * (g + w);
}

// One warp per block: lane l holds cells l and l + 32 (rows l / 8 and l / 8 + 4,
// column l % 8), and the block's 32 ghosts are one a lane (face l / 8, position
// l % 8 along it).  A warp's loads of a block, its own cells and its ghosts, go
// out together (the faces' table entries are read one block ahead), and the
// stencil's neighbours come by shuffles: no shared memory, no CTA barrier, so
// an SM keeps all its warps' loads in flight.  Four blocks to a CTA with labs in
// shared memory waited at a CTA barrier for the slowest ghost's dependent loads;
// labs of one warp each were bound by the L1/shared-memory pipe (79-86 % busy,
// lab rows and interleaved pairs conflicting).  us on 1.15 M blocks (73 M cells),
// CTA labs -> warp labs -> shuffles: right-hand side and the reset of pres 1833
// -> 1686 -> 1393, correction 1028 -> 724 -> 585; on 0.1 M blocks 225 -> 206 -> 172 and
// 127 -> 89 -> 77.  With the ghosts' operands of all fields loaded together
// (Ghost::values) 1139 (4.1 TB/s) and 462 (6.3 TB/s) on 1.15 M blocks.  Bound now by
// the ghosts' scattered sectors.

// The neighbours of a lane's two values a0 (cell l), a1 (cell l + 32): across
// the block's faces the ghosts g of the other lanes.
struct Around {
  double w[2], e[2], s[2], n[2];
};
__device__ __forceinline__ double from_lane(double v, int src) { return __shfl_sync(kFull, v, src & 31); }

__device__ __forceinline__ void around_x(int lane, double a0, double a1, double g, Around& o) {
  const int r = lane >> 3, c = lane & 7;
  const int src = c == 7 ? 8 + r : r;  // column 0 takes the W ghosts of its rows, column 7 the E ghosts
  const double g0 = from_lane(g, src), g1 = from_lane(g, src + 4);
  const double w0 = from_lane(a0, lane - 1), w1 = from_lane(a1, lane - 1);
  const double e0 = from_lane(a0, lane + 1), e1 = from_lane(a1, lane + 1);
  o.w[0] = c > 0 ? w0 : g0;
  o.w[1] = c > 0 ? w1 : g1;
  o.e[0] = c < 7 ? e0 : g0;
  o.e[1] = c < 7 ? e1 : g1;
}
__device__ __forceinline__ void around_y(int lane, double a0, double a1, double g, Around& o) {
  const int r = lane >> 3, c = lane & 7;
  const double gg = from_lane(g, (r == 3 ? 24 : 16) + c);  // row 0 takes the S ghosts, row 7 the N ghosts
  const double n0 = from_lane(a0, lane + 8), n1 = from_lane(a1, lane + 8);
  const double s0 = from_lane(a0, lane - 8), s1 = from_lane(a1, lane - 8);
  o.s[0] = r > 0 ? s0 : gg;
  o.n[0] = r < 3 ? n0 : n1;  // row 3 -> row 4
  o.s[1] = r > 0 ? s1 : s0;  // row 4 -> row 3
  o.n[1] = r < 3 ? n1 : gg;
}

// Whether each of a block's faces has finer neighbours (bit f), from its
// lanes' sides.
__device__ __forceinline__ unsigned finer_faces(int kind) {
  const unsigned m = __ballot_sync(kFull, kind == kFiner);
  return (m & 1u) | ((m >> 7) & 2u) | ((m >> 14) & 4u) | ((m >> 21) & 8u);
}

// The flux corrections (one a ghost lane, on finer faces) at a lane's two
// cells: across x (faces W, E) and across y (face S of cell l, N of cell l + 32).
struct FluxAt {
  double x[2], y;
  bool w, e, s, n;
  __device__ __forceinline__ FluxAt(int lane, unsigned finer, double corr) {
    const int r = lane >> 3, c = lane & 7;
    const int src = c == 7 ? 8 + r : r;
    x[0] = from_lane(corr, src);
    x[1] = from_lane(corr, src + 4);
    y = from_lane(corr, (r == 3 ? 24 : 16) + c);
    w = c == 0 && (finer & 1u);
    e = c == 7 && (finer & 2u);
    s = r == 0 && (finer & 4u);
    n = r == 3 && (finer & 8u);
  }
};

// VEL, PRES: which of the two right-hand side parts the call asks for.
template <bool VEL, bool PRES>
__global__ void __launch_bounds__(kProjThreads, 3) k_pressure_rhs(const __grid_constant__ Geo G, double dt,
                                                                    const __grid_constant__ ProjFields P) {
  const int lane = threadIdx.x & 31;
  const int f = lane >> 3;
  const int64_t step = (int64_t)gridDim.x * kProjWarps;
  int64_t b = (int64_t)blockIdx.x * kProjWarps + (threadIdx.x >> 5);
  int32_t code = 0, level = 0;
  if (b < G.F.nb) {
    code = __ldg(G.nbr + 4 * b + f);
    level = __ldg(G.F.level + b);
  }
  for (; b < G.F.nb; b += step) {
    const int64_t cell = b * kBLEN + lane;
    double2 u[2], ud[2];
    double chi[2], p[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      if constexpr (VEL) {
        u[j] = __ldg(reinterpret_cast<const double2*>(P.vel) + cell + 32 * j);
        ud[j] = __ldg(reinterpret_cast<const double2*>(P.udef) + cell + 32 * j);
        chi[j] = __ldg(P.chi + cell + 32 * j);
      }
      if constexpr (PRES) p[j] = P.pres[cell + 32 * j];
    }
    const Ghost gh(G, b, lane, G.side_from_code(b, f, code));
    const unsigned finer = finer_faces(gh.s.kind);
    const double h = cell_h(G.F, level);
    const double facDiv = 0.5 * h / dt;
    const int cmp = gh.xface() ? 0 : 1;  // the normal component: the only one the divergence reads
    FaceVals v[3];  // vel, udef (VEL), pres (PRES)
    if constexpr (VEL && PRES) {
      const Fld w[3] = {{P.vel, 2, cmp, true}, {P.udef, 2, cmp, true}, {P.pres, 1, 0, false}};
      gh.values(w, v);
    } else if constexpr (VEL) {
      const Fld w[2] = {{P.vel, 2, cmp, true}, {P.udef, 2, cmp, true}};
      gh.values(w, reinterpret_cast<FaceVals(&)[2]>(v));
    } else {
      const Fld w[1] = {{P.pres, 1, 0, false}};
      gh.values(w, reinterpret_cast<FaceVals(&)[1]>(v[2]));
    }
    // the next block's faces
    const int64_t bn = b + step;
    if (bn < G.F.nb) {
      code = __ldg(G.nbr + 4 * bn + f);
      level = __ldg(G.F.level + bn);
    }
    double corr[2] = {0.0, 0.0};  // flux corrections: divergence, Laplacian
    if (gh.s.kind == kFiner) {
      if constexpr (VEL) {
        int64_t fb;
        int k0;
        gh.fine_cells(fb, k0);
        const double chif[2] = {__ldg(P.chi + gh.fine_cell(fb, k0, 0, 0)), __ldg(P.chi + gh.fine_cell(fb, k0, 1, 0))};
        const double own = div_face(f, facDiv, __ldg(P.chi + gh.cell), v[0].g, v[0].own, v[1].g, v[1].own);
        const double facDivF = 0.5 * (0.5 * h) / dt;  // the finer blocks' h: half, exactly
        double fs[2];
#pragma unroll
        for (int r = 0; r < 2; ++r)
          fs[r] = div_face(f ^ 1, facDivF, chif[r], v[0].fine_ghost[r], v[0].fine[r], v[1].fine_ghost[r], v[1].fine[r]);
        corr[0] = own + (fs[0] + fs[1]);
      }
      if constexpr (PRES) {
        const double own = v[2].g - v[2].own;
        double fs[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) fs[r] = v[2].fine_ghost[r] - v[2].fine[r];
        corr[1] = own + (fs[0] + fs[1]);
      }
    }
    __syncwarp();
    double t[2];
    if constexpr (VEL) {
      Around a, d;
      around_x(lane, u[0].x, u[1].x, v[0].g, a);
      around_y(lane, u[0].y, u[1].y, v[0].g, a);
      around_x(lane, ud[0].x, ud[1].x, v[1].g, d);
      around_y(lane, ud[0].y, ud[1].y, v[1].g, d);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        t[j] = facDiv * ((a.e[j] - a.w[j]) + (a.n[j] - a.s[j]));
        t[j] += -facDiv * chi[j] * ((d.e[j] - d.w[j]) + (d.n[j] - d.s[j]));
      }
      if (finer) {  // in face order
        const FluxAt q(lane, finer, corr[0]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (q.w) t[j] = t[j] + q.x[j];
          if (q.e) t[j] = t[j] + q.x[j];
        }
        if (q.s) t[0] = t[0] + q.y;
        if (q.n) t[1] = t[1] + q.y;
      }
    } else {
      t[0] = P.tmp[cell];
      t[1] = P.tmp[cell + 32];
    }
    if constexpr (PRES) {
      Around a;
      around_x(lane, p[0], p[1], v[2].g, a);
      around_y(lane, p[0], p[1], v[2].g, a);
#pragma unroll
      for (int j = 0; j < 2; ++j) t[j] -= ((a.w[j] + a.e[j]) + (a.s[j] + a.n[j])) - 4.0 * p[j];
      if (finer) {
        const FluxAt q(lane, finer, corr[1]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (q.w) t[j] = t[j] + q.x[j];
          if (q.e) t[j] = t[j] + q.x[j];
        }
        if (q.s) t[0] = t[0] + q.y;
        if (q.n) t[1] = t[1] + q.y;
      }
      P.pold[cell] = p[0];
      P.pold[cell + 32] = p[1];
    }
    P.tmp[cell] = t[0];
    P.tmp[cell + 32] = t[1];
  }
}

__global__ void __launch_bounds__(kProjThreads, 4) k_pressure_correction(const __grid_constant__ Geo G, double dt,
                                                                           const double* __restrict__ pres,
                                                                           double* __restrict__ vel) {
  const int lane = threadIdx.x & 31;
  const Fld Q[1] = {{pres, 1, 0, false}};
  const int f = lane >> 3;
  const int64_t step = (int64_t)gridDim.x * kProjWarps;
  int64_t b = (int64_t)blockIdx.x * kProjWarps + (threadIdx.x >> 5);
  int32_t code = 0, level = 0;
  if (b < G.F.nb) {
    code = __ldg(G.nbr + 4 * b + f);
    level = __ldg(G.F.level + b);
  }
  for (; b < G.F.nb; b += step) {
    const int64_t cell = b * kBLEN + lane;
    const double p[2] = {__ldg(pres + cell), __ldg(pres + cell + 32)};
    double2 v[2];  // updated in place: no read-only path
#pragma unroll
    for (int j = 0; j < 2; ++j) v[j] = reinterpret_cast<const double2*>(vel)[cell + 32 * j];
    const Ghost gh(G, b, lane, G.side_from_code(b, f, code));
    const unsigned finer = finer_faces(gh.s.kind);
    const double h = cell_h(G.F, level);
    const double pFac = -0.5 * dt * h;
    FaceVals q[1];
    gh.values(Q, q);
    const double g = q[0].g;
    const int64_t bn = b + step;
    if (bn < G.F.nb) {
      code = __ldg(G.nbr + 4 * bn + f);
      level = __ldg(G.F.level + bn);
    }
    double corr = 0.0;
    if (gh.s.kind == kFiner) {
      const double own = grad_face(f, pFac, g, q[0].own);
      const double pFacF = -0.5 * dt * (0.5 * h);  // the finer blocks' h: half, exactly
      double fs[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) fs[r] = grad_face(f ^ 1, pFacF, q[0].fine_ghost[r], q[0].fine[r]);
      corr = own + (fs[0] + fs[1]);
    }
    __syncwarp();
    Around a;
    around_x(lane, p[0], p[1], g, a);
    around_y(lane, p[0], p[1], g, a);
    double tx[2], ty[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      tx[j] = pFac * (a.e[j] - a.w[j]);
      ty[j] = pFac * (a.n[j] - a.s[j]);
    }
    if (finer) {
      const FluxAt q(lane, finer, corr);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (q.w) tx[j] = tx[j] + q.x[j];
        if (q.e) tx[j] = tx[j] + q.x[j];
      }
      if (q.s) ty[0] = ty[0] + q.y;
      if (q.n) ty[1] = ty[1] + q.y;
    }
    const double ih2 = 1.0 / h / h;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      v[j].x += tx[j] * ih2;
      v[j].y += ty[j] * ih2;
      reinterpret_cast<double2*>(vel)[cell + 32 * j] = v[j];
    }
  }
}

// Persistent grid: the co-resident CTAs of a kernel (queried once per device).
int persistent_grid(const void* fn, int which, int64_t ngroups) {
  static std::atomic<int> cap[64][4];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int g = cap[dev][which].load(std::memory_order_acquire);
  if (g <= 0) {
    int sms = 0, per_sm = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kProjThreads, 0) != cudaSuccess)
      return 0;
    g = std::max(1, sms * per_sm);
    cap[dev][which].store(g, std::memory_order_release);
  }
  return (int)std::min<int64_t>(g, ngroups);
}

}  // namespace

cudaError_t launch_pressure_rhs(const ForestView& F, const int32_t* nbr, double dt, const ProjFields& f,
                                cudaStream_t s) {
  if (F.nb <= 0) return cudaSuccess;
  const int which = (f.vel ? 2 : 0) + (f.pres ? 1 : 0);
  if (which == 0) return cudaErrorInvalidValue;
  auto* const fn = which == 3 ? k_pressure_rhs<true, true> : which == 2 ? k_pressure_rhs<true, false>
                                                                        : k_pressure_rhs<false, true>;
  const int grid = persistent_grid((const void*)fn, which, (F.nb + kProjWarps - 1) / kProjWarps);
  if (grid <= 0) return cudaErrorInvalidConfiguration;
  fn<<<grid, kProjThreads, 0, s>>>(Geo{F, nbr}, dt, f);
  return cudaGetLastError();
}

cudaError_t launch_pressure_correction(const ForestView& F, const int32_t* nbr, double dt, const double* pres,
                                       double* vel, cudaStream_t s) {
  if (F.nb <= 0) return cudaSuccess;
  const int grid = persistent_grid((const void*)k_pressure_correction, 0, (F.nb + kProjWarps - 1) / kProjWarps);
  if (grid <= 0) return cudaErrorInvalidConfiguration;
  k_pressure_correction<<<grid, kProjThreads, 0, s>>>(Geo{F, nbr}, dt, pres, vel);
  return cudaGetLastError();
}

}  // namespace cup2d
