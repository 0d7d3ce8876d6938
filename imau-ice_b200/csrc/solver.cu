// solver.cu -- the linear solve of solve_DIVA_stag_linearised
// (ice_velocity_module.f90:1656-1761), which the reference assembles as a CSR
// matrix (rows :1762-2589) and hands to PETSc KSP or SOR
// (utilities_module.f90:600-718, petsc_module.F90:23-90).
//
// Here the matrix is never formed.  The operator is applied matrix-free from
// N_a, N_b and beta_eff (the coefficients of the reference's free rows,
// :2342-2467), and the domain-boundary rows (:1932-2191: u - u_in = 0,
// u = 0, u - u_opp = 0) are eliminated exactly: a boundary unknown is read
// through its source (the inner or opposite unknown, or zero), so only
// interior unknowns are solved for and the boundary values are filled from
// them afterwards.  The solver is BiCGStab, right-preconditioned with one
// geometric-multigrid V-cycle:
//   * levels coarsen the a-grid by 2 in each direction with at least 9 points
//     (semi-coarsening once one direction is small), so cells may become
//     anisotropic; the coarse operator is the same staggered discretisation
//     rediscretised on the coarse grid with cell aspect hy/hx and averaged
//     N_a, N_b, beta_eff;
//   * transfers are bilinear on the staggered u (cx) and v (cy) points,
//     restriction = transpose of prolongation;
//   * smoothing is 4-colour Gauss-Seidel (u red/black, v red/black), with the
//     exact diagonal of the reduced system;
//   * the larger levels are smoothed by tile kernels, the largest of them in streamed strips
//     (halo recomputed instead of exchanged; two launches per level and V-cycle, three for a
//     streamed level below the finest, whose right-hand side is restricted first), the coarse
//     levels whose data fit in 200 KB run out of one thread block's shared memory (one launch
//     per V-cycle), and the coarsest level is solved directly with its inverse, formed once per
//     viscosity iteration, or relaxed where it has none.
// All reductions are two-stage (block partials, then one fixed-order sum) so
// results are bit-reproducible from run to run.
#include <cmath>
#include <cstdio>
#include <algorithm>
#include <utility>
#include <vector>
#include "ctx.hpp"
#include "wave_geom.hpp"

namespace diva {
namespace {

#ifndef DIVA_SUB_THREADS
#define DIVA_SUB_THREADS 1024
#endif
constexpr int kSubThreads = DIVA_SUB_THREADS;   // threads of the one-block coarse-level kernel

// A level's operator.  R is the type of its coefficients and of the x values it is
// applied to: double everywhere, float for the finest level's smoother copies of the
// mixed-precision preconditioner (precision = DIVA_PREC_MIXED).
template <class R>
struct OpT {
  Dims d;
  BCs bc;
  double ax, ay;   // hy/hx and hx/hy of the level's cells (1 on the fine grid)
  const R *Na, *Nb, *Bx, *By;
  // 'BC' ice margins (finest level only, else null): the type of each u and v row
  const int8_t *rtu, *rtv;
  double inv_dx;
};
using Op = OpT<double>;

// Row types of the finest level with choice_ice_margin 'BC' (solve_DIVA_stag_linearised
// :1683-1727): a free row, u = 0 (shelf next to land, or a front cell with ocean on both
// sides), or the calving-front stress row of list_DIVA_matrix_coefficients_eq_1_margin
// (:2192-2266) / eq_2_margin (:2267-2341) with the ice on the lower (west/south) or upper
// side of the face.
enum : int8_t { RT_FREE = 0, RT_IDENT = 1, RT_MARGIN_LO = 2, RT_MARGIN_HI = 3 };

__host__ __device__ __forceinline__ bool u_int(const Dims& d, int j, int i) {
  return i >= 1 && i <= d.nx - 3 && j >= 1 && j <= d.ny - 2;
}
__host__ __device__ __forceinline__ bool v_int(const Dims& d, int j, int i) {
  return i >= 1 && i <= d.nx - 2 && j >= 1 && j <= d.ny - 3;
}
__host__ __device__ __forceinline__ int bc_pick(int a, int b) {
  if (a == DIVA_BC_ZERO || b == DIVA_BC_ZERO) return DIVA_BC_ZERO;
  if (a == DIVA_BC_INFINITE || b == DIVA_BC_INFINITE) return DIVA_BC_INFINITE;
  return DIVA_BC_PERIODIC;
}
// Source of u(j,i) (list_DIVA_matrix_coefficients_eq_1_boundary :1932-2061); false = zero.
__host__ __device__ __forceinline__ bool u_src(const Dims& d, const BCs& b, int j, int i, int& js, int& is) {
  if (u_int(d, j, i)) { js = j; is = i; return true; }
  const bool W = i == 0, E = i == d.nx - 2, S = j == 0, N = j == d.ny - 1;
  int t;
  if (W && S) t = bc_pick(b.uS, b.uW);
  else if (E && S) t = bc_pick(b.uS, b.uE);
  else if (W && N) t = bc_pick(b.uN, b.uW);
  else if (E && N) t = bc_pick(b.uN, b.uE);
  else if (W) t = b.uW;
  else if (E) t = b.uE;
  else if (S) t = b.uS;
  else t = b.uN;
  if (t == DIVA_BC_ZERO) return false;
  if (t == DIVA_BC_INFINITE) { is = W ? 1 : (E ? d.nx - 3 : i); js = S ? 1 : (N ? d.ny - 2 : j); }
  else { is = W ? d.nx - 3 : (E ? 1 : i); js = S ? d.ny - 2 : (N ? 1 : j); }
  return true;
}
// Source of v(j,i) (list_DIVA_matrix_coefficients_eq_2_boundary :2062-2191).
__host__ __device__ __forceinline__ bool v_src(const Dims& d, const BCs& b, int j, int i, int& js, int& is) {
  if (v_int(d, j, i)) { js = j; is = i; return true; }
  const bool W = i == 0, E = i == d.nx - 1, S = j == 0, N = j == d.ny - 2;
  int t;
  if (W && S) t = bc_pick(b.vS, b.vW);
  else if (E && S) t = bc_pick(b.vS, b.vE);
  else if (W && N) t = bc_pick(b.vN, b.vW);
  else if (E && N) t = bc_pick(b.vN, b.vE);
  else if (W) t = b.vW;
  else if (E) t = b.vE;
  else if (S) t = b.vS;
  else t = b.vN;
  if (t == DIVA_BC_ZERO) return false;
  if (t == DIVA_BC_INFINITE) { is = W ? 1 : (E ? d.nx - 2 : i); js = S ? 1 : (N ? d.ny - 3 : j); }
  else { is = W ? d.nx - 2 : (E ? 1 : i); js = S ? d.ny - 3 : (N ? 1 : j); }
  return true;
}
// Where the x values of the (j,i) point live: a full plane of the level (GIx), or
// a shared-memory tile whose origin is (j0,i0) and whose rows hold rj points (TIx).
struct GIx {
  Dims d;
  __device__ __forceinline__ long long operator()(int j, int i) const { return d.at(j, i); }
};
struct TIx {
  int j0, i0, rj;
  __device__ __forceinline__ int operator()(int j, int i) const { return (i - i0) * rj + (j - j0); }
};

// Read a u (v) value through the boundary elimination (RAW = false), or as
// stored (RAW = true: the reference's assembled rows reference stored values).
template <bool RAW, class R, class IX>
__device__ __forceinline__ R LUx(const OpT<R>& o, const R* x, const IX& ix, int j, int i) {
  if (RAW) return x[ix(j, i)];
  int js, is;
  return u_src(o.d, o.bc, j, i, js, is) ? x[ix(js, is)] : R(0);
}
template <bool RAW, class R, class IX>
__device__ __forceinline__ R LVx(const OpT<R>& o, const R* x, const IX& ix, int j, int i) {
  if (RAW) return x[ix(j, i)];
  int js, is;
  return v_src(o.d, o.bc, j, i, js, is) ? x[ix(js, is)] : R(0);
}
template <bool RAW = false>
__device__ __forceinline__ double LU(const Op& o, const double* x, int j, int i) {
  return LUx<RAW>(o, x, GIx{o.d}, j, i);
}
template <bool RAW = false>
__device__ __forceinline__ double LV(const Op& o, const double* x, int j, int i) {
  return LVx<RAW>(o, x, GIx{o.d}, j, i);
}

// Sum of the nine stencil terms, accumulated with explicit fused multiply-adds in a
// fixed order, so every code path of a level (boundary-mapped reads, plain reads, tiles, the
// ring) rounds identically whatever the compiler would contract.
__device__ __forceinline__ double fma_r(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fma_r(float a, float b, float c) { return fmaf(a, b, c); }

template <class R>
__device__ __forceinline__ R stencil9(R c0, R x0, R c1, R x1, R c2, R x2, R c3, R x3, R c4, R x4, R c5, R x5, R c6,
                                      R x6, R c7, R x7, R c8, R x8) {
  R s = c0 * x0;
  s = fma_r(c1, x1, s);
  s = fma_r(c2, x2, s);
  s = fma_r(c3, x3, s);
  s = fma_r(c4, x4, s);
  s = fma_r(c5, x5, s);
  s = fma_r(c6, x6, s);
  s = fma_r(c7, x7, s);
  return fma_r(c8, x8, s);
}

template <class R>
__device__ __forceinline__ R stencil4(R c0, R x0, R c1, R x1, R c2, R x2, R c3, R x3) {
  R s = c0 * x0;
  s = fma_r(c1, x1, s);
  s = fma_r(c2, x2, s);
  return fma_r(c3, x3, s);
}

// (A x) of the u row at interior (j,i) (list_DIVA_matrix_coefficients_eq_1_free :2342-2404)
// IX places x values, CX the coefficients N_a, N_b, B (a level plane or a shared-memory tile)
// (the constants are written R(k) so that R = double performs exactly the double
// operations of the reference's rows and R = float stays in single precision)
template <bool RAW, bool FRONT = true, class R, class IX, class CX>
__device__ __forceinline__ R AuXC(const OpT<R>& o, const R* xu, const R* xv, const IX& ix, const CX& cx, int j,
                                  int i) {
  if (FRONT && o.rtu) {
    const int t = o.rtu[o.d.at(j, i)];
    if (t == RT_IDENT) return xu[ix(j, i)];
    if (t != RT_FREE) {   // front row: -4N u(i1-1) + 4N u(i1) - 2N v(j-1,i1) + 2N v(j,i1), N = N_a(i1)/dx
      const int i1 = t == RT_MARGIN_LO ? i : i + 1;
      const R N = o.Na[cx(j, i1)], idx = R(o.inv_dx);
      return stencil4(R(-4) * idx * N, LUx<RAW>(o, xu, ix, j, i1 - 1), R(4) * idx * N, LUx<RAW>(o, xu, ix, j, i1),
                      R(-2) * idx * N, LVx<RAW>(o, xv, ix, j - 1, i1), R(2) * idx * N, LVx<RAW>(o, xv, ix, j, i1));
    }
  }
  const R Ae = o.Na[cx(j, i + 1)], Aw = o.Na[cx(j, i)], Bn = o.Nb[cx(j, i)], Bs = o.Nb[cx(j - 1, i)];
  const R ax = R(o.ax), ay = R(o.ay);
  const R cE = R(4) * ax * Ae, cW = R(4) * ax * Aw, cN = ay * Bn, cS = ay * Bs;
  const R diag = -(cE + cW + cN + cS) - o.Bx[cx(j, i)];
  return stencil9(cE, LUx<RAW>(o, xu, ix, j, i + 1), cW, LUx<RAW>(o, xu, ix, j, i - 1), cN,
                  LUx<RAW>(o, xu, ix, j + 1, i), cS, LUx<RAW>(o, xu, ix, j - 1, i), diag, xu[ix(j, i)],
                  R(-2) * Aw - Bn, LVx<RAW>(o, xv, ix, j, i), R(2) * Ae + Bn, LVx<RAW>(o, xv, ix, j, i + 1),
                  R(2) * Aw + Bs, LVx<RAW>(o, xv, ix, j - 1, i), R(-2) * Ae - Bs, LVx<RAW>(o, xv, ix, j - 1, i + 1));
}
// (A x) of the v row at interior (j,i) (list_DIVA_matrix_coefficients_eq_2_free :2405-2467)
template <bool RAW, bool FRONT = true, class R, class IX, class CX>
__device__ __forceinline__ R AvXC(const OpT<R>& o, const R* xu, const R* xv, const IX& ix, const CX& cx, int j,
                                  int i) {
  if (FRONT && o.rtv) {
    const int t = o.rtv[o.d.at(j, i)];
    if (t == RT_IDENT) return xv[ix(j, i)];
    if (t != RT_FREE) {   // front row: -4N v(j1-1) + 4N v(j1) - 2N u(j1,i-1) + 2N u(j1,i), N = N_a(j1)/dx
      const int j1 = t == RT_MARGIN_LO ? j : j + 1;
      const R N = o.Na[cx(j1, i)], idx = R(o.inv_dx);
      return stencil4(R(-4) * idx * N, LVx<RAW>(o, xv, ix, j1 - 1, i), R(4) * idx * N, LVx<RAW>(o, xv, ix, j1, i),
                      R(-2) * idx * N, LUx<RAW>(o, xu, ix, j1, i - 1), R(2) * idx * N, LUx<RAW>(o, xu, ix, j1, i));
    }
  }
  const R An = o.Na[cx(j + 1, i)], As = o.Na[cx(j, i)], Be = o.Nb[cx(j, i)], Bw = o.Nb[cx(j, i - 1)];
  const R ax = R(o.ax), ay = R(o.ay);
  const R cN = R(4) * ay * An, cS = R(4) * ay * As, cE = ax * Be, cW = ax * Bw;
  const R diag = -(cN + cS + cE + cW) - o.By[cx(j, i)];
  return stencil9(cN, LVx<RAW>(o, xv, ix, j + 1, i), cS, LVx<RAW>(o, xv, ix, j - 1, i), cE,
                  LVx<RAW>(o, xv, ix, j, i + 1), cW, LVx<RAW>(o, xv, ix, j, i - 1), diag, xv[ix(j, i)],
                  R(-2) * An - Bw, LUx<RAW>(o, xu, ix, j + 1, i - 1), R(2) * An + Be, LUx<RAW>(o, xu, ix, j + 1, i),
                  R(2) * As + Bw, LUx<RAW>(o, xu, ix, j, i - 1), R(-2) * As - Be, LUx<RAW>(o, xu, ix, j, i));
}
template <bool RAW, class IX>
__device__ __forceinline__ double AuX(const Op& o, const double* xu, const double* xv, const IX& ix, int j, int i) {
  return AuXC<RAW>(o, xu, xv, ix, GIx{o.d}, j, i);
}
template <bool RAW, class IX>
__device__ __forceinline__ double AvX(const Op& o, const double* xu, const double* xv, const IX& ix, int j, int i) {
  return AvXC<RAW>(o, xu, xv, ix, GIx{o.d}, j, i);
}
template <bool RAW = false>
__device__ __forceinline__ double Au(const Op& o, const double* xu, const double* xv, int j, int i) {
  return AuX<RAW>(o, xu, xv, GIx{o.d}, j, i);
}
template <bool RAW = false>
__device__ __forceinline__ double Av(const Op& o, const double* xu, const double* xv, int j, int i) {
  return AvX<RAW>(o, xu, xv, GIx{o.d}, j, i);
}
// effective diagonal of the reduced system: couplings to boundary unknowns whose source is the row itself fold in
__device__ __forceinline__ double diag_u(const Op& o, int j, int i) {
  const Dims& d = o.d;
  if (o.rtu) {
    const int t = o.rtu[d.at(j, i)];
    if (t == RT_IDENT) return 1.0;
    if (t != RT_FREE) {   // the u terms of the front row whose source is this row
      const int i1 = t == RT_MARGIN_LO ? i : i + 1;
      const double N = o.Na[d.at(j, i1)];
      double dg = 0.0;
      int js, is;
      if (u_src(d, o.bc, j, i1 - 1, js, is) && js == j && is == i) dg += -4.0 * o.inv_dx * N;
      if (u_src(d, o.bc, j, i1, js, is) && js == j && is == i) dg += 4.0 * o.inv_dx * N;
      return dg;
    }
  }
  const double Ae = o.Na[d.at(j, i + 1)], Aw = o.Na[d.at(j, i)], Bn = o.Nb[d.at(j, i)], Bs = o.Nb[d.at(j - 1, i)];
  const double cE = 4.0 * o.ax * Ae, cW = 4.0 * o.ax * Aw, cN = o.ay * Bn, cS = o.ay * Bs;
  double dg = -(cE + cW + cN + cS) - o.Bx[d.at(j, i)];
  int js, is;
  if (!u_int(d, j, i + 1) && u_src(d, o.bc, j, i + 1, js, is) && js == j && is == i) dg += cE;
  if (!u_int(d, j, i - 1) && u_src(d, o.bc, j, i - 1, js, is) && js == j && is == i) dg += cW;
  if (!u_int(d, j + 1, i) && u_src(d, o.bc, j + 1, i, js, is) && js == j && is == i) dg += cN;
  if (!u_int(d, j - 1, i) && u_src(d, o.bc, j - 1, i, js, is) && js == j && is == i) dg += cS;
  return dg;
}
__device__ __forceinline__ double diag_v(const Op& o, int j, int i) {
  const Dims& d = o.d;
  if (o.rtv) {
    const int t = o.rtv[d.at(j, i)];
    if (t == RT_IDENT) return 1.0;
    if (t != RT_FREE) {
      const int j1 = t == RT_MARGIN_LO ? j : j + 1;
      const double N = o.Na[d.at(j1, i)];
      double dg = 0.0;
      int js, is;
      if (v_src(d, o.bc, j1 - 1, i, js, is) && js == j && is == i) dg += -4.0 * o.inv_dx * N;
      if (v_src(d, o.bc, j1, i, js, is) && js == j && is == i) dg += 4.0 * o.inv_dx * N;
      return dg;
    }
  }
  const double An = o.Na[d.at(j + 1, i)], As = o.Na[d.at(j, i)], Be = o.Nb[d.at(j, i)], Bw = o.Nb[d.at(j, i - 1)];
  const double cN = 4.0 * o.ay * An, cS = 4.0 * o.ay * As, cE = o.ax * Be, cW = o.ax * Bw;
  double dg = -(cN + cS + cE + cW) - o.By[d.at(j, i)];
  int js, is;
  if (!v_int(d, j + 1, i) && v_src(d, o.bc, j + 1, i, js, is) && js == j && is == i) dg += cN;
  if (!v_int(d, j - 1, i) && v_src(d, o.bc, j - 1, i, js, is) && js == j && is == i) dg += cS;
  if (!v_int(d, j, i + 1) && v_src(d, o.bc, j, i + 1, js, is) && js == j && is == i) dg += cE;
  if (!v_int(d, j, i - 1) && v_src(d, o.bc, j, i - 1, js, is) && js == j && is == i) dg += cW;
  return dg;
}

#define IDX2D                                                            \
  const int j = blockIdx.x * blockDim.x + threadIdx.x;                   \
  const int i = blockIdx.y * blockDim.y + threadIdx.y;

// Gauss-Seidel update of one point of one component (comp 0 = u, 1 = v).  Every smoother
// (these per-colour kernels, the tiles, the streamed kernel, the sub-cycle) forms x + (b - A x) / diag as one
// explicit fused multiply-add; those of one level also sum a row's terms in one order, so they
// round alike.
__device__ __forceinline__ void gs_point(const Op& o, double* xu, double* xv, const double* bu, const double* bv,
                                         const double* idu, const double* idv, int comp, int j, int i) {
  const long long q = o.d.at(j, i);
  if (comp == 0) {
    if (u_int(o.d, j, i)) xu[q] = fma(bu[q] - Au(o, xu, xv, j, i), idu[q], xu[q]);
  } else {
    if (v_int(o.d, j, i)) xv[q] = fma(bv[q] - Av(o, xu, xv, j, i), idv[q], xv[q]);
  }
}

// one colour of Gauss-Seidel: comp 0 = u, 1 = v; colour = (i+j) parity
__global__ void k_gs(Op o, double* xu, double* xv, const double* bu, const double* bv, const double* idu,
                     const double* idv, int comp, int color) {
  const int jj = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = blockIdx.y * blockDim.y + threadIdx.y;
  const int j = 2 * jj + ((i + color) & 1);
  if (j >= o.d.ny || i >= o.d.nx) return;
  gs_point(o, xu, xv, bu, bv, idu, idv, comp, j, i);
}

// r = b - A x on the interior (zero elsewhere)
__device__ __forceinline__ void residual_point(const Op& o, const double* xu, const double* xv, const double* bu,
                                               const double* bv, double* ru, double* rv, int j, int i) {
  const long long q = o.d.at(j, i);
  ru[q] = u_int(o.d, j, i) ? bu[q] - Au(o, xu, xv, j, i) : 0.0;
  rv[q] = v_int(o.d, j, i) ? bv[q] - Av(o, xu, xv, j, i) : 0.0;
}
__global__ void k_residual(Op o, const double* xu, const double* xv, const double* bu, const double* bv, double* ru,
                           double* rv) {
  IDX2D
  if (j >= o.d.ny || i >= o.d.nx) return;
  residual_point(o, xu, xv, bu, bv, ru, rv, j, i);
}

// 1D transfer weights.  "cell" direction: u along x, v along y; "node": u along y, v along x.
// Gather form of the restriction: coarse C collects fine f with weight w; tap k of at most
// 4 (cell) or 3 (node), or the single tap f = C, w = 1 where the level is not coarsened
// along that direction (f2 = 1).  The taps are formed in registers, one at a time, and
// summed with explicit fused multiply-adds (the weights' products are exact), so every
// kernel that restricts or prolongs rounds alike.
__host__ __device__ __forceinline__ int gather_cell_n(int f2) { return f2 == 1 ? 1 : 4; }
__host__ __device__ __forceinline__ int gather_node_n(int f2) { return f2 == 1 ? 1 : 3; }
__host__ __device__ __forceinline__ void gather_cell(int C, int f2, int k, int& f, double& w) {
  if (f2 == 1) { f = C; w = 1.0; return; }
  f = 2 * C - 1 + k; w = (k == 0 || k == 3) ? 0.25 : 0.75;
}
__host__ __device__ __forceinline__ void gather_node(int C, int f2, int k, int& f, double& w) {
  if (f2 == 1) { f = C; w = 1.0; return; }
  f = 2 * C - 1 + k; w = k == 1 ? 1.0 : 0.5;
}
// Scatter form (prolongation): fine f takes coarse C with weight w; tap k of at most 2.
__host__ __device__ __forceinline__ int scatter_cell_n(int f, int f2) { return f2 == 1 ? 1 : 2; }
__host__ __device__ __forceinline__ int scatter_node_n(int f, int f2) { return f2 == 1 ? 1 : ((f & 1) == 0 ? 1 : 2); }
__host__ __device__ __forceinline__ void scatter_cell(int f, int f2, int k, int& C, double& w) {
  if (f2 == 1) { C = f; w = 1.0; return; }
  const int c = f >> 1;
  C = k == 0 ? c : ((f & 1) == 0 ? c - 1 : c + 1);
  w = k == 0 ? 0.75 : 0.25;
}
__host__ __device__ __forceinline__ void scatter_node(int f, int f2, int k, int& C, double& w) {
  if (f2 == 1) { C = f; w = 1.0; return; }
  const int c = f >> 1;
  if ((f & 1) == 0) { C = c; w = 1.0; return; }
  C = c + k; w = 0.5;
}

// b_c = P^T r_f on coarse interior points; x_c = 0
// (P^T r_f) at the coarse point (j,i): the restricted u and v residuals (zero off the coarse interior)
template <class RR>
__device__ __forceinline__ void restrict_values(const Dims& df, const Dims& dc, int fx, int fy, const RR* ru,
                                                const RR* rv, int j, int i, double& bu, double& bv) {
  double s = 0.0;
  if (u_int(dc, j, i)) {
    const int ni = gather_cell_n(fx), nj = gather_node_n(fy);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (a >= nj) break;
      int fj; double wj;
      gather_node(j, fy, a, fj, wj);
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        if (b >= ni) break;
        int fi; double wi;
        gather_cell(i, fx, b, fi, wi);
        if (u_int(df, fj, fi)) s = fma(wj * wi, (double)ru[df.at(fj, fi)], s);
      }
    }
  }
  bu = s;
  s = 0.0;
  if (v_int(dc, j, i)) {
    const int ni = gather_node_n(fx), nj = gather_cell_n(fy);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      if (a >= nj) break;
      int fj; double wj;
      gather_cell(j, fy, a, fj, wj);
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        if (b >= ni) break;
        int fi; double wi;
        gather_node(i, fx, b, fi, wi);
        if (v_int(df, fj, fi)) s = fma(wj * wi, (double)rv[df.at(fj, fi)], s);
      }
    }
  }
  bv = s;
}
// b_c = P^T r_f on coarse interior points; x_c = 0
__device__ __forceinline__ void restrict_point(const Dims& df, const Dims& dc, int fx, int fy, const double* ru,
                                               const double* rv, double* bu, double* bv, double* xu, double* xv,
                                               int j, int i) {
  const long long q = dc.at(j, i);
  restrict_values(df, dc, fx, fy, ru, rv, j, i, bu[q], bv[q]);
  xu[q] = 0.0;
  xv[q] = 0.0;
}
__global__ void k_restrict(Dims df, Dims dc, int fx, int fy, const double* ru, const double* rv, double* bu,
                           double* bv, double* xu, double* xv) {
  IDX2D
  if (j >= dc.ny || i >= dc.nx) return;
  restrict_point(df, dc, fx, fy, ru, rv, bu, bv, xu, xv, j, i);
}

// P x_c at the fine point (j,i): increments of u and v (coarse values read through the
// coarse boundary mapping); zero off the fine interior
__device__ __forceinline__ void prolong_delta(const Op& oc, const Dims& df, int fx, int fy, const double* xcu,
                                              const double* xcv, int j, int i, double& du, double& dv) {
  const Dims& dc = oc.d;
  du = 0.0;
  dv = 0.0;
  if (u_int(df, j, i)) {
    const int ni = scatter_cell_n(i, fx), nj = scatter_node_n(j, fy);
    double s = 0.0;
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      if (a >= nj) break;
      int Cj; double wj;
      scatter_node(j, fy, a, Cj, wj);
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        if (b >= ni) break;
        int Ci; double wi;
        scatter_cell(i, fx, b, Ci, wi);
        const int J = min(max(Cj, 0), dc.ny - 1), I = min(max(Ci, 0), dc.nx - 2);
        s = fma(wj * wi, LU(oc, xcu, J, I), s);
      }
    }
    du = s;
  }
  if (v_int(df, j, i)) {
    const int ni = scatter_node_n(i, fx), nj = scatter_cell_n(j, fy);
    double s = 0.0;
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      if (a >= nj) break;
      int Cj; double wj;
      scatter_cell(j, fy, a, Cj, wj);
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        if (b >= ni) break;
        int Ci; double wi;
        scatter_node(i, fx, b, Ci, wi);
        const int J = min(max(Cj, 0), dc.ny - 2), I = min(max(Ci, 0), dc.nx - 1);
        s = fma(wj * wi, LV(oc, xcv, J, I), s);
      }
    }
    dv = s;
  }
}
// P x_c at the fine point (j,i) of a level coarsened by 2 in both directions, from the
// coarse correction staged in shared memory: cu/cv hold, for the coarse region whose
// origin is (CJ0,CI0) (CRJ rows per column), the values prolong_delta reads (the clamped
// position read through the coarse boundary mapping).  The same taps, weights and order.
__device__ __forceinline__ void prolong_delta_staged(const Dims& df, const double* cu, const double* cv, int CJ0,
                                                     int CI0, int CRJ, int j, int i, double& du, double& dv) {
  du = 0.0;
  dv = 0.0;
  if (u_int(df, j, i)) {
    const int ni = scatter_cell_n(i, 2), nj = scatter_node_n(j, 2);
    double s = 0.0;
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      if (a >= nj) break;
      int Cj; double wj;
      scatter_node(j, 2, a, Cj, wj);
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        if (b >= ni) break;
        int Ci; double wi;
        scatter_cell(i, 2, b, Ci, wi);
        s = fma(wj * wi, cu[(Ci - CI0) * CRJ + (Cj - CJ0)], s);
      }
    }
    du = s;
  }
  if (v_int(df, j, i)) {
    const int ni = scatter_node_n(i, 2), nj = scatter_cell_n(j, 2);
    double s = 0.0;
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      if (a >= nj) break;
      int Cj; double wj;
      scatter_cell(j, 2, a, Cj, wj);
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        if (b >= ni) break;
        int Ci; double wi;
        scatter_node(i, 2, b, Ci, wi);
        s = fma(wj * wi, cv[(Ci - CI0) * CRJ + (Cj - CJ0)], s);
      }
    }
    dv = s;
  }
}
// x_f += P x_c on fine interior points
__device__ __forceinline__ void prolong_point(const Op& oc, const Dims& df, int fx, int fy, const double* xcu,
                                              const double* xcv, double* xu, double* xv, int j, int i) {
  const long long q = df.at(j, i);
  double du, dv;
  prolong_delta(oc, df, fx, fy, xcu, xcv, j, i, du, dv);
  if (u_int(df, j, i)) xu[q] += du;
  if (v_int(df, j, i)) xv[q] += dv;
}
__global__ void k_prolong(Op oc, Dims df, int fx, int fy, const double* xcu, const double* xcv, double* xu,
                          double* xv) {
  IDX2D
  if (j >= df.ny || i >= df.nx) return;
  prolong_point(oc, df, fx, fy, xcu, xcv, xu, xv, j, i);
}

// ---- tiled smoothing of the large levels ---------------------------------------------
// One block owns a TJ x TI tile of a level and keeps x and b of the tile plus a
// halo of H points on every side in shared memory (H = 4 nu + 1 for nu sweeps per
// phase: kHalo for two, kHaloOne for one).  Colour pass q of a smoothing phase
// updates the points within H-1-q of the tile.  Every value
// a row reads -- its stencil neighbours and, on an 'infinite' or 'zero' side, the
// inner point a boundary unknown is mapped to -- lies within one point of the row,
// so after the 8 passes of V(2,2)'s pre- or post-smoothing the tile and one ring
// around it hold exactly what the level-wide colour sweeps produce, and the
// residual of the tile follows from them.  The halo is recomputed by the
// neighbouring blocks instead of exchanged.  A periodic side maps a boundary
// unknown across the domain, so such grids use the per-colour kernels.
constexpr int kHalo = 9;        // the widest halo: 2 sweeps (8 colour passes) + 1
constexpr int kHaloOne = 5;     // the halo of 1 sweep (4 colour passes) + 1
constexpr int kTileThreads = 512;
// the halo a tile kernel needs for `sweeps` smoothing sweeps per phase
inline int halo_for(int sweeps) { return sweeps <= 1 ? kHaloOne : kHalo; }

// STAGE: the region's coefficients (N_a, N_b, B_x, B_y and the inverse diagonals)
// are staged in shared memory too, so the colour passes touch no global memory.
// R: the type of the tile's values and coefficients (float on the finest level of the
// mixed-precision preconditioner, else double).
template <int TJ, int TI, bool STAGE, class R = double, int H = kHalo>
struct TileGeom {
  static constexpr int RJ = TJ + 2 * H, RI = TI + 2 * H, N = RJ * RI;
  static constexpr size_t smem = (STAGE ? 10 : 4) * N * sizeof(R);   // x, b (+ 6 coefficient planes)
  // the post-smoothing kernel also stages the coarse correction under its region (a
  // level coarsened by 2 in both directions): CRJ x CRI coarse points, u and v, in double
  static constexpr int CRJ = RJ / 2 + 3, CRI = RI / 2 + 3;
  static constexpr size_t coarse_off = (smem + 7) / 8;   // in doubles
  static constexpr size_t smem_up = (coarse_off + 2 * CRJ * CRI) * sizeof(double);
};

// A block whose whole region lies in the interior of both components (u: 1 <= i <=
// nx-3, 1 <= j <= ny-2; v: 1 <= i <= nx-2, 1 <= j <= ny-3) reads every stencil value
// as stored: the boundary mapping is the identity there, so DEEP blocks skip it and
// the interior tests (the same values, decided once per block).
constexpr bool kTileDeepPath = true;
template <int TJ, int TI, int H>
__device__ __forceinline__ bool tile_deep(const TIx& ix, const Dims& d) {
  constexpr int RJ = TJ + 2 * H, RI = TI + 2 * H;
  return kTileDeepPath && ix.i0 >= 1 && ix.i0 + RI - 1 <= d.nx - 3 && ix.j0 >= 1 && ix.j0 + RJ - 1 <= d.ny - 3;
}

// The shared-memory planes of a tile kernel and the operator reading from them.
// FRONT: the operator may carry 'BC' front rows (only the finest level's kernels with
// choice_ice_margin 'BC'); without it the row-type test is compiled out.
template <int TJ, int TI, bool STAGE, bool FRONT, class R, int H>
struct TileMem {
  R *xu, *xv, *bu, *bv;
  const R *iu, *iv;   // inverse diagonals: staged plane or the level's
  OpT<R> os;          // the level's operator, coefficients staged when STAGE
  __device__ TileMem(R* sm, const OpT<R>& o, const R* idu, const R* idv) {
    using G = TileGeom<TJ, TI, STAGE, R, H>;
    xu = sm; xv = sm + G::N; bu = sm + 2 * G::N; bv = sm + 3 * G::N;
    os = o;
    iu = idu; iv = idv;
    if (STAGE) {
      os.Na = sm + 4 * G::N; os.Nb = sm + 5 * G::N; os.Bx = sm + 6 * G::N; os.By = sm + 7 * G::N;
      iu = sm + 8 * G::N; iv = sm + 9 * G::N;
    }
  }
  // stage the region's coefficients (out-of-domain points are never read)
  __device__ void stage(const OpT<R>& o, const R* idu, const R* idv, const TIx& ix, int t, bool in, long long q) {
    if (!STAGE) return;
    using G = TileGeom<TJ, TI, STAGE, R, H>;
    R* sm = xu;
    sm[4 * G::N + t] = in ? o.Na[q] : R(0);
    sm[5 * G::N + t] = in ? o.Nb[q] : R(0);
    sm[6 * G::N + t] = in ? o.Bx[q] : R(0);
    sm[7 * G::N + t] = in ? o.By[q] : R(0);
    sm[8 * G::N + t] = in ? idu[q] : R(0);
    sm[9 * G::N + t] = in ? idv[q] : R(0);
  }
  template <bool RAW>
  __device__ __forceinline__ R Au(const TIx& ix, int j, int i) const {
    if (STAGE) return AuXC<RAW, FRONT>(os, xu, xv, ix, ix, j, i);
    return AuXC<RAW, FRONT>(os, xu, xv, ix, GIx{os.d}, j, i);
  }
  template <bool RAW>
  __device__ __forceinline__ R Av(const TIx& ix, int j, int i) const {
    if (STAGE) return AvXC<RAW, FRONT>(os, xu, xv, ix, ix, j, i);
    return AvXC<RAW, FRONT>(os, xu, xv, ix, GIx{os.d}, j, i);
  }
  __device__ __forceinline__ R idu(const TIx& ix, int j, int i) const {
    return STAGE ? iu[ix(j, i)] : iu[os.d.at(j, i)];
  }
  __device__ __forceinline__ R idv(const TIx& ix, int j, int i) const {
    return STAGE ? iv[ix(j, i)] : iv[os.d.at(j, i)];
  }
  // Boundary unknowns in the tile ("ghosts").  A u or v value outside its component's
  // interior is read, by the rows next to it, through the boundary elimination (u_src,
  // v_src): as the value of its source point, or as zero.  The tile keeps each such value
  // in its own slot, equal to its source's value, so every row of a block reads its whole
  // stencil as stored, at the domain's edge too.  The elimination maps a row's outside
  // same-component neighbours back to the row itself (read before the row's own update),
  // and cross-component ghosts are read only in the other component's passes, so a
  // component's ghosts are refreshed from their sources (ghost_refresh) after the staging
  // and after each pair of that component's colour passes: every read then sees the value
  // the elimination would read.  (Periodic sides, whose sources lie across the
  // domain, do not use the tiles.)
  __device__ __forceinline__ bool in_region(const TIx& ix, int j, int i) const {
    using G = TileGeom<TJ, TI, STAGE, R, H>;
    return j >= ix.j0 && j < ix.j0 + G::RJ && i >= ix.i0 && i < ix.i0 + G::RI;
  }
  // The new value of the interior u point (j,i) into the ghosts whose source it is: by
  // u_src's rule, the edge point beyond it on an 'infinite' side and the corner beyond it
  // where two such sides meet.
  __device__ __forceinline__ void ghosts_u(const TIx& ix, int j, int i, R val) {
    const Dims& d = os.d;
    const BCs& b = os.bc;
    const bool W = i == 1, E = i == d.nx - 3, S = j == 1, N = j == d.ny - 2;
    if (!(W || E || S || N)) return;
    auto put = [&](int jg, int ig) { if (in_region(ix, jg, ig)) xu[ix(jg, ig)] = val; };
    constexpr int INF = DIVA_BC_INFINITE;
    if (W && b.uW == INF) put(j, 0);
    if (E && b.uE == INF) put(j, d.nx - 2);
    if (S && b.uS == INF) put(0, i);
    if (N && b.uN == INF) put(d.ny - 1, i);
    if (W && S && bc_pick(b.uS, b.uW) == INF) put(0, 0);
    if (E && S && bc_pick(b.uS, b.uE) == INF) put(0, d.nx - 2);
    if (W && N && bc_pick(b.uN, b.uW) == INF) put(d.ny - 1, 0);
    if (E && N && bc_pick(b.uN, b.uE) == INF) put(d.ny - 1, d.nx - 2);
  }
  // Every source point of the region (the interior points on the lines i = 1, the last
  // interior column, j = 1 and the last interior row of each component) writes its current
  // value into its ghosts; one point per thread.
  __device__ __forceinline__ void ghost_refresh(const TIx& ix, int comps = 3) {   // bit 0: u, bit 1: v
    using G = TileGeom<TJ, TI, STAGE, R, H>;
    const Dims& d = os.d;
    // the four lines of each component, clipped to the region: 2 vertical (RJ points each)
    // and 2 horizontal (RI points each)
    const int per = 2 * G::RJ + 2 * G::RI;
    const int t0 = (comps & 1) ? 0 : per, t1 = (comps & 2) ? 2 * per : per;
    for (int t = t0 + threadIdx.x; t < t1; t += blockDim.x) {
      const bool ucomp = t < per;
      const int e = ucomp ? t : t - per;
      int j, i;
      if (e < 2 * G::RJ) {   // a column line: i = 1 or the last interior column
        j = ix.j0 + e % G::RJ;
        i = e < G::RJ ? 1 : (ucomp ? d.nx - 3 : d.nx - 2);
      } else {               // a row line: j = 1 or the last interior row
        const int f = e - 2 * G::RJ;
        i = ix.i0 + f % G::RI;
        j = f < G::RI ? 1 : (ucomp ? d.ny - 2 : d.ny - 3);
      }
      if (!in_region(ix, j, i)) continue;
      if (ucomp) {
        if (u_int(d, j, i)) ghosts_u(ix, j, i, xu[ix(j, i)]);
      } else {
        if (v_int(d, j, i)) ghosts_v(ix, j, i, xv[ix(j, i)]);
      }
    }
  }
  // the same for the interior v point (j,i) (v_src's rule)
  __device__ __forceinline__ void ghosts_v(const TIx& ix, int j, int i, R val) {
    const Dims& d = os.d;
    const BCs& b = os.bc;
    const bool W = i == 1, E = i == d.nx - 2, S = j == 1, N = j == d.ny - 3;
    if (!(W || E || S || N)) return;
    auto put = [&](int jg, int ig) { if (in_region(ix, jg, ig)) xv[ix(jg, ig)] = val; };
    constexpr int INF = DIVA_BC_INFINITE;
    if (W && b.vW == INF) put(j, 0);
    if (E && b.vE == INF) put(j, d.nx - 1);
    if (S && b.vS == INF) put(0, i);
    if (N && b.vN == INF) put(d.ny - 2, i);
    if (W && S && bc_pick(b.vS, b.vW) == INF) put(0, 0);
    if (E && S && bc_pick(b.vS, b.vE) == INF) put(0, d.nx - 1);
    if (W && N && bc_pick(b.vN, b.vW) == INF) put(d.ny - 2, 0);
    if (E && N && bc_pick(b.vN, b.vE) == INF) put(d.ny - 2, d.nx - 1);
  }
};

// one colour pass over the region points within `reach` of the tile
template <bool DEEP, class M>
__device__ __forceinline__ void tile_pass(M& m, const TIx& ix, int TJ, int TI, int tj0, int ti0, int comp, int color,
                                          int reach) {
  const Dims& d = m.os.d;
  // the box of points within `reach` of the tile, one colour of it
  const int bj0 = tj0 - reach, bi0 = ti0 - reach, BJ = TJ + 2 * reach, BI = TI + 2 * reach;
  const int hj = (BJ + 1) / 2;
  for (int t = threadIdx.x; t < hj * BI; t += blockDim.x) {
    const int i = bi0 + t / hj;
    const int j = bj0 + 2 * (t % hj) + ((color + i + bj0) & 1);   // (i + j) & 1 == color
    if (j >= bj0 + BJ) continue;
    if (!DEEP && (j < 0 || j >= d.ny || i < 0 || i >= d.nx)) continue;
    const int k = ix(j, i);
    // every stencil value is read as stored: at the domain's edge the ghosts hold what
    // the boundary elimination would read
    if (comp == 0) {
      if (DEEP || u_int(d, j, i)) m.xu[k] = fma_r(m.bu[k] - m.template Au<true>(ix, j, i), m.idu(ix, j, i), m.xu[k]);
    } else {
      if (DEEP || v_int(d, j, i)) m.xv[k] = fma_r(m.bv[k] - m.template Av<true>(ix, j, i), m.idv(ix, j, i), m.xv[k]);
    }
  }
}
template <int TJ, int TI, class M>
__device__ __forceinline__ void tile_pass_any(bool deep, M& m, const TIx& ix, int tj0, int ti0, int comp, int color,
                                              int reach) {
  if (deep) tile_pass<true>(m, ix, TJ, TI, tj0, ti0, comp, color, reach);
  else tile_pass<false>(m, ix, TJ, TI, tj0, ti0, comp, color, reach);
}

// Source of b for a pre-smoothing kernel: given on the level (the finest), or the
// restriction of the finer level's residual, computed where it is needed.
struct Restriction {
  int on;              // 0: b given in gbu/gbv
  Dims df;             // finer level
  int fx, fy;          // coarsening factors from it
  const void *ru, *rv; // its residual: double, or float (rfloat) from a mixed-precision finest level
  int rfloat;
};
__device__ __forceinline__ void restrict_from(const Restriction& rs, const Dims& dc, int j, int i, double& b0,
                                              double& b1) {
  if (rs.rfloat)
    restrict_values(rs.df, dc, rs.fx, rs.fy, static_cast<const float*>(rs.ru), static_cast<const float*>(rs.rv), j,
                    i, b0, b1);
  else
    restrict_values(rs.df, dc, rs.fx, rs.fy, static_cast<const double*>(rs.ru), static_cast<const double*>(rs.rv),
                    j, i, b0, b1);
}

// pre-smoothing from x = 0 (the descent of a V-cycle enters every level with x = 0):
// `sweeps` forward sweeps (u0 u1 v0 v1), then x, b and r = b - A x of the tile.
// b is read (and, when restricted here, stored) in double; x and r are written in R.
template <int TJ, int TI, bool STAGE, bool FRONT, class R, int H>
__global__ void __launch_bounds__(kTileThreads) k_smooth_down(OpT<R> o, Restriction rs, double* gbu, double* gbv,
                                                              R* gxu, R* gxv, R* gru, R* grv, const R* idu,
                                                              const R* idv, int sweeps) {
  constexpr int RJ = TJ + 2 * H, N = RJ * (TI + 2 * H);
  extern __shared__ double smd[];
  R* sm = reinterpret_cast<R*>(smd);
  TileMem<TJ, TI, STAGE, FRONT, R, H> m(sm, o, idu, idv);
  const Dims& d = o.d;
  const int tj0 = blockIdx.x * TJ, ti0 = blockIdx.y * TI;
  const TIx ix{tj0 - H, ti0 - H, RJ};
  const bool deep = tile_deep<TJ, TI, H>(ix, d);
  for (int t = threadIdx.x; t < N; t += blockDim.x) {
    const int j = ix.j0 + t % RJ, i = ix.i0 + t / RJ;
    const bool in = j >= 0 && j < d.ny && i >= 0 && i < d.nx;
    const long long q = in ? d.at(j, i) : 0;
    double b0 = 0.0, b1 = 0.0;
    if (in) {
      if (rs.on) {
        restrict_from(rs, d, j, i, b0, b1);
      } else {
        b0 = gbu[q];
        b1 = gbv[q];
      }
    }
    m.xu[t] = R(0);
    m.xv[t] = R(0);
    m.bu[t] = R(b0);
    m.bv[t] = R(b1);
    m.stage(o, idu, idv, ix, t, in, q);
  }
  __syncthreads();
  int pass = 0;
  for (int s = 0; s < sweeps; ++s)
    for (int p = 0; p < 4; ++p, ++pass) {
      tile_pass_any<TJ, TI>(deep, m, ix, tj0, ti0, p >> 1, p & 1, H - 1 - pass);
      __syncthreads();
      if (!deep && (p & 1)) {   // a component's pair done: its ghosts from their sources
        m.ghost_refresh(ix, 1 << (p >> 1));
        __syncthreads();
      }
    }
  for (int t = threadIdx.x; t < TJ * TI; t += blockDim.x) {
    const int j = tj0 + t % TJ, i = ti0 + t / TJ;
    if (j >= d.ny || i >= d.nx) continue;
    const long long q = d.at(j, i);
    const int k = ix(j, i);
    gxu[q] = m.xu[k];
    gxv[q] = m.xv[k];
    if (rs.on) {
      gbu[q] = m.bu[k];
      gbv[q] = m.bv[k];
    }
    if (deep) {
      gru[q] = m.bu[k] - m.template Au<true>(ix, j, i);
      grv[q] = m.bv[k] - m.template Av<true>(ix, j, i);
    } else {
      // the ghosts hold the boundary values: stored reads
      gru[q] = u_int(d, j, i) ? m.bu[k] - m.template Au<true>(ix, j, i) : R(0);
      grv[q] = v_int(d, j, i) ? m.bv[k] - m.template Av<true>(ix, j, i) : R(0);
    }
  }
}

// post-smoothing: x += P x_c, then `sweeps` backward sweeps (v1 v0 u1 u0); x of the tile.
// The pre-smoothed x is read over the halo from (gxu, gxv) and the result written to
// (oxu, oxv): separate arrays, since blocks of other tiles may still be reading the
// halo when this block writes (the grid runs in several waves on large levels).  The
// coarse correction and b are double; the smoothing runs in R; the output is double.
template <int TJ, int TI, bool STAGE, bool FRONT, class R, int H>
__global__ void __launch_bounds__(kTileThreads) k_smooth_up(OpT<R> o, Op oc, int fx, int fy, const double* xcu,
                                                            const double* xcv, const double* gbu, const double* gbv,
                                                            const R* gxu, const R* gxv, double* oxu, double* oxv,
                                                            const R* idu, const R* idv, int sweeps) {
  constexpr int RJ = TJ + 2 * H, N = RJ * (TI + 2 * H);
  extern __shared__ double smd[];
  R* sm = reinterpret_cast<R*>(smd);
  TileMem<TJ, TI, STAGE, FRONT, R, H> m(sm, o, idu, idv);
  const Dims& d = o.d;
  const int tj0 = blockIdx.x * TJ, ti0 = blockIdx.y * TI;
  const TIx ix{tj0 - H, ti0 - H, RJ};
  const bool deep = tile_deep<TJ, TI, H>(ix, d);
  // The coarse correction under the region, staged once (a level coarsened by 2 in both
  // directions): each coarse value is read from L2 once per block instead of by every
  // fine point that takes it (up to 8 reads per fine point).
  using G = TileGeom<TJ, TI, STAGE, R, H>;
  const bool staged = fx == 2 && fy == 2;
  const int CJ0 = (ix.j0 >> 1) - 1, CI0 = (ix.i0 >> 1) - 1;
  double* cu = smd + G::coarse_off;
  double* cv = cu + G::CRJ * G::CRI;
  if (staged) {
    const Dims& dc = oc.d;
    for (int t = threadIdx.x; t < G::CRJ * G::CRI; t += blockDim.x) {
      const int J = CJ0 + t % G::CRJ, I = CI0 + t / G::CRJ;
      cu[t] = LU(oc, xcu, min(max(J, 0), dc.ny - 1), min(max(I, 0), dc.nx - 2));
      cv[t] = LV(oc, xcv, min(max(J, 0), dc.ny - 2), min(max(I, 0), dc.nx - 1));
    }
    __syncthreads();
  }
  for (int t = threadIdx.x; t < N; t += blockDim.x) {
    const int j = ix.j0 + t % RJ, i = ix.i0 + t / RJ;
    const bool in = j >= 0 && j < d.ny && i >= 0 && i < d.nx;
    const long long q = in ? d.at(j, i) : 0;
    double xa = 0.0, xb = 0.0, ba = 0.0, bb = 0.0;
    if (in) {
      double du, dv;
      if (staged) prolong_delta_staged(d, cu, cv, CJ0, CI0, G::CRJ, j, i, du, dv);
      else prolong_delta(oc, d, fx, fy, xcu, xcv, j, i, du, dv);
      xa = gxu[q];
      xb = gxv[q];
      if (u_int(d, j, i)) xa += du;
      if (v_int(d, j, i)) xb += dv;
      ba = gbu[q];
      bb = gbv[q];
    }
    m.xu[t] = R(xa);
    m.xv[t] = R(xb);
    m.bu[t] = R(ba);
    m.bv[t] = R(bb);
    m.stage(o, idu, idv, ix, t, in, q);
  }
  __syncthreads();
  if (!deep) {
    // The ghosts take their sources' staged values: every interior point on the lines next
    // to the domain's edge writes its own ghosts (ghosts_u/ghosts_v), so only those
    // lines are visited.  A 'zero' ghost holds 0 already (the pre-smoothing left it so).
    m.ghost_refresh(ix);
    __syncthreads();
  }
  int pass = 0;
  for (int s = 0; s < sweeps; ++s)
    for (int p = 3; p >= 0; --p, ++pass) {
      tile_pass_any<TJ, TI>(deep, m, ix, tj0, ti0, p >> 1, p & 1, H - 1 - pass);
      __syncthreads();
      if (!deep && !(p & 1)) {   // a component's pair done: its ghosts from their sources
        m.ghost_refresh(ix, 1 << (p >> 1));
        __syncthreads();
      }
    }
  for (int t = threadIdx.x; t < TJ * TI; t += blockDim.x) {
    const int j = tj0 + t % TJ, i = ti0 + t / TJ;
    if (j >= d.ny || i >= d.nx) continue;
    const long long q = d.at(j, i);
    const int k = ix(j, i);
    oxu[q] = (deep || u_int(d, j, i)) ? (double)m.xu[k] : 0.0;   // no ghost values out
    oxv[q] = (deep || v_int(d, j, i)) ? (double)m.xv[k] : 0.0;
  }
}

// ---- streamed smoothing of the large levels --------------------------------------------
// One block owns a strip of rows (j) and a chunk of columns (i) of a level and sweeps over the
// chunk two columns a step.  A ring of columns in shared memory holds x, b and the operator's
// coefficients of the columns in flight; colour pass q of a smoothing phase runs 3 q columns
// behind the first, each pass in a warp of its own, so that in every step all passes (and the
// copies of the columns ahead, the prolongation and the output) work on different columns and
// one barrier separates the steps:
//   step s: copy the pair s + kWavePre, prolong columns 2 s and 2 s + 1, pass q on columns
//           2 s - 3 - 3 q and the next, output columns 2 s - 3 - 3 NP and the next.
// A pass reads its columns and the two beside them.  With three columns between consecutive
// passes every value it reads has been through exactly the passes of the level-wide colour
// sweeps: pass q - 1 left the column beyond one step ago, pass q + 1 reaches the column before
// one step from now (the two columns' points of one colour do not read each other).  The halo
// (H = NP + 1 points: one per pass and one for the residual) is recomputed by the neighbouring
// blocks instead of exchanged, at the ends of the chunk and along the strip's sides, pass q
// updating the points within H - 1 - q of the tile.  The columns arrive by bulk copies (one
// per plane and column) that complete on mbarriers.
//
// Bound by latency: a step lasts as long as one point update (nine reads, 30 dependent operations,
// a write) and its barrier; the schedulers issue in half of the cycles, shared memory is busy in a
// fifth (counters at 321 x 561).  A colour's points in one column lie two rows apart, a 2-way bank
// conflict; half of a half-warp takes the column's points and the other half the next column's,
// whose rows have the other parity, so the 16 values fill all banks.
// Against the square tiles (k_smooth_down/up), which recompute 9 points on every side and keep
// no more than 32 x 32 points and no coefficients beside them: a strip's halo along i is paid
// once per chunk, and the coefficients come from the ring.  Pre- and post-smoothing of the
// 1501 x 1501 sheet 312 us (tiles 408), of the 321 x 561 cap 48 us (tiles 53); a step of two
// columns takes 0.7 us, most of it the latency of one point update after the other.  Issuing
// the columns as tensor copies of two columns by one thread was slower (379 us).
//
// Boundary unknowns ("ghosts"): a u or v value outside its component's interior is read, by
// the rows next to it, as its source's value or as zero (u_src, v_src).  The ring keeps each
// such value in its own slot; the thread that updates a source point writes its ghosts as
// well, so every row reads its whole stencil as stored.  (Corner ghosts are read by no
// interior row.  Periodic sides, whose sources lie across the domain, use the per-colour
// kernels.)
struct WaveArgs {
  Op o;
  const double *idu, *idv;
  const double *bu, *bv;
  double *xu, *xv;            // pre-smoothed x: written by the descent, read by the ascent
  double *ru, *rv;            // descent: the residual
  double *ou, *ov;       // ascent: the result
  Op oc;                 // ascent: the coarser level and its correction
  const double *xcu, *xcv;
  int fx, fy;
  int rows, chunk;       // tile height and width
  double* fail;          // set when a wait ran out
  int drop;              // issue no copies, so that the waits run out (tests)
};

// ring offsets of the three columns a row reads
struct RIx {
  int w, c, e, i, j0;
  __device__ __forceinline__ int operator()(int jj, int ii) const {
    return (ii == i ? c : (ii > i ? e : w)) + (jj - j0);
  }
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool wave_wait(uint32_t bar, uint32_t parity) {
  for (int it = 0; it < kWaveSpin; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// Where a coarse column position is read from along i: clamped, then through the boundary rule
// (u: cx points, v: cy points); rows are mapped by the reader.  -1: zero everywhere.
__device__ __forceinline__ int coarse_col(const Op& oc, int C, bool ucomp) {
  const int last = ucomp ? oc.d.nx - 2 : oc.d.nx - 1;
  const int I = min(max(C, 0), last);
  const int west = ucomp ? oc.bc.uW : oc.bc.vW, east = ucomp ? oc.bc.uE : oc.bc.vE;
  if (I == 0) return west == DIVA_BC_INFINITE ? 1 : -1;
  if (I == last) return east == DIVA_BC_INFINITE ? last - 1 : -1;
  return I;
}

// Two taps of the prolongation along one direction, C and weight (the second weight 0 where
// there is one tap: adding 0 x keeps the sum's bits).
__device__ __forceinline__ void two_taps(int f, int fac, bool cell, int (&C)[2], double (&w)[2]) {
  const int n = cell ? scatter_cell_n(f, fac) : scatter_node_n(f, fac);
  if (cell) scatter_cell(f, fac, 0, C[0], w[0]);
  else scatter_node(f, fac, 0, C[0], w[0]);
  C[1] = C[0];
  w[1] = 0.0;
  if (n == 2) {
    if (cell) scatter_cell(f, fac, 1, C[1], w[1]);
    else scatter_node(f, fac, 1, C[1], w[1]);
  }
}

// Every role runs its own loop over the steps, with ring offsets that move on by one column a
// step: the step lasts as long as its slowest warp, so each warp's instructions count.
template <bool FRONT, bool UP>
__global__ void __launch_bounds__(32 * (UP ? WaveGeom::warps_up : WaveGeom::warps_down))
    k_wave(const __grid_constant__ WaveArgs a) {
  using G = WaveGeom;
  constexpr int NP = G::NP, H = G::H, RP = G::RP, NC = G::NC, CP = G::CP, COL = 8 * RP;
  constexpr int NPW = G::passes, NOUT = UP ? G::out_up : G::out_down;
  extern __shared__ __align__(128) unsigned char wsm[];
  __shared__ __align__(8) uint64_t bars[kWaveBars];
  double* ring = reinterpret_cast<double*>(wsm);                          // [NC][8: xu xv Na Nb Bx By idu idv][RP]
  double* bring = reinterpret_cast<double*>(wsm + G::xk);        // [NC][2][RP]
  double* cring = reinterpret_cast<double*>(wsm + G::xk + G::b); // [kWaveCoarse][2][CP]
  const Dims& d = a.o.d;
  const BCs& bc = a.o.bc;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tj0 = blockIdx.x * a.rows, ti0 = blockIdx.y * a.chunk;
  const int j0 = tj0 - G::HB, i0 = ti0 - H;                      // the ring's first row, the region's first column
  const int tw = min(a.chunk, d.nx - ti0), ncols = tw + 2 * H;   // tile width here, region columns
  const int CJ0 = a.fy == 2 ? ((j0 >> 1) - 2) & ~1 : j0 - 2;     // first coarse row held (even)
  const int last = (tw + H + 3 * NP + 2) / 2;   // the step that puts out the tile's last column
  constexpr int kINF = DIVA_BC_INFINITE;

  if (threadIdx.x == 0) {
    for (int k = 0; k < kWaveBars; ++k)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&bars[k])), "r"(kWaveCopy) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  // the operator reading from the ring
  Op os = a.o;
  os.Na = ring + 2 * RP; os.Nb = ring + 3 * RP; os.Bx = ring + 4 * RP; os.By = ring + 5 * RP;
  auto slot_of = [](int cc) { return ((cc % NC) + NC) % NC * COL; };
  auto next2 = [](int off) { return off >= (NC - 2) * COL ? off - (NC - 2) * COL : off + 2 * COL; };
  auto beside = [&](int off, int i) {   // the three columns around ring offset off
    return RIx{off == 0 ? (NC - 1) * COL : off - COL, off, off == (NC - 1) * COL ? 0 : off + COL, i, j0};
  };
  // a new value of the interior point (j,i) into the ghosts whose source it is (x: its plane;
  // il, jl: the last interior column and row)
  auto ghosts = [&](double* x, const RIx& ix, int j, int i, int il, int jl, int gW, int gE, int gS, int gN, double val) {
    if (gS == kINF && j == 1) x[ix.c - j0] = val;
    if (gN == kINF && j == jl) x[ix.c + jl + 1 - j0] = val;
    if (gW == kINF && i == 1) x[ix.w + j - j0] = val;
    if (gE == kINF && i == il) x[ix.e + j - j0] = val;
  };

  if (warp < NPW) {
    // ---- pass q: lanes 0-7, 16-23 the first column's points, 8-15, 24-31 the second's
    const int q = warp >> 1, p4 = q & 3, p = UP ? 3 - p4 : p4, comp = p >> 1, color = p & 1, reach = H - 1 - q;
    const int il = comp == 0 ? d.nx - 3 : d.nx - 2, jl = comp == 0 ? d.ny - 2 : d.ny - 3;   // interior 1 .. il, 1 .. jl
    const int jlo = tj0 - reach, jmin = max(jlo, 1), jmax = min(tj0 + a.rows + reach - 1, jl);
    const int c0 = max(H - reach, 1 - i0), c1 = min(H + tw + reach - 1, il - i0);           // region columns updated
    const int gW = comp == 0 ? bc.uW : bc.vW, gE = comp == 0 ? bc.uE : bc.vE;
    const int gS = comp == 0 ? bc.uS : bc.vS, gN = comp == 0 ? bc.uN : bc.vN;
    double* x = ring + comp * RP;
    const double* xu = ring;
    const double* xv = ring + RP;
    const double* id = ring + (6 + comp) * RP;
    const double* bb = bring + comp * RP;
    int cc = -3 - 3 * q + ((lane >> 3) & 1), off = slot_of(cc);
    // (i + j) & 1 == color: a lane's column keeps its parity
    const int j = jlo + ((color + i0 + cc + jlo) & 1) + 2 * ((lane & 7) | ((lane >> 4) << 3)) + 32 * (warp & 1);
    const bool row = j >= jmin && j <= jmax, jghost = j == 1 || j == jl;
    __syncthreads();   // the first columns are there
#pragma unroll 1
    for (int s = 0; s <= last; ++s, cc += 2, off = next2(off)) {
      if (row && cc >= c0 && cc <= c1) {
        const int i = i0 + cc;
        const RIx ix = beside(off, i);
        const int k = off + j - j0;
        const double b = bb[(off >> 2) + j - j0];   // (the b ring has a quarter of the planes)
        const double Ax = comp == 0 ? AuXC<true, FRONT>(os, xu, xv, ix, ix, j, i) : AvXC<true, FRONT>(os, xu, xv, ix, ix, j, i);
        const double val = fma_r(b - Ax, id[k], x[k]);
        x[k] = val;
        if (jghost || i == 1 || i == il) ghosts(x, ix, j, i, il, jl, gW, gE, gS, gN, val);
      }
      __syncthreads();
    }
  } else if (warp < NPW + NOUT) {
    // ---- the tile's values
    const int w = warp - NPW, comp = UP ? 0 : w >> 2, h0 = UP ? 0 : (w >> 1) & 1, jj = (w & 1) * 32 + lane, j = tj0 + jj;
    const bool row = jj < a.rows && j < d.ny;
    const double* xu = ring;
    const double* xv = ring + RP;
    int cc = -3 - 3 * NP + h0, off = slot_of(cc);
    __syncthreads();
#pragma unroll 1
    for (int s = 0; s <= last; ++s, cc += 2, off = next2(off)) {
      int o = off;
#pragma unroll
      for (int h = 0; h < (UP ? 2 : 1); ++h) {
        const int c = cc + h, i = i0 + c, k = o + j - j0;
        if (c >= H && c < H + tw && row) {
          const long long g = d.at(j, i);
          if (UP) {   // no ghost values out
            a.ou[g] = u_int(d, j, i) ? xu[k] : 0.0;
            a.ov[g] = v_int(d, j, i) ? xv[k] : 0.0;
          } else {
            const RIx ix = beside(o, i);
            const double b = bring[(o >> 2) + comp * RP + j - j0];
            if (comp == 0) {
              a.xu[g] = xu[k];
              a.ru[g] = u_int(d, j, i) ? b - AuXC<true, FRONT>(os, xu, xv, ix, ix, j, i) : 0.0;
            } else {
              a.xv[g] = xv[k];
              a.rv[g] = v_int(d, j, i) ? b - AvXC<true, FRONT>(os, xu, xv, ix, ix, j, i) : 0.0;
            }
          }
        }
        o = o == (NC - 1) * COL ? 0 : o + COL;
      }
      __syncthreads();
    }
  } else if (warp < NPW + NOUT + kWaveCopy) {
    // ---- copies of pair s + kWavePre: copy c = 5 w + lane of 20 is plane c / 2 of column c % 2; the
    // last warp moves the coarse columns (lane 0: u, 1: v), or zeroes x for the descent
    const int w = warp - NPW - NOUT, copy = min(5 * w + lane, 19), pl = copy >> 1, hc = copy & 1;
    const bool mover = w < kWaveCopy - 1;
    const int r0 = max(0, -j0), r1 = min(RP, d.ld - j0);           // ring rows inside the planes (even numbers)
    const int cr0 = max(0, -CJ0), cr1 = UP ? min(CP, a.oc.d.ld - CJ0) : 0;
    constexpr uint32_t es = sizeof(double);
    const uint32_t bytes = mover && lane < 5 && (UP || pl >= 2) && r1 > r0 ? (r1 - r0) * es : 0;
    uint32_t sum[2] = {hc == 0 ? bytes : 0, hc == 1 ? bytes : 0};  // the warp's bytes of either column
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      sum[0] += __shfl_down_sync(0xffffffffu, sum[0], o);          // (lanes 0-7 to lane 0)
      sum[1] += __shfl_down_sync(0xffffffffu, sum[1], o);
    }
    const void* plane = pl == 0 ? (const void*)a.xu : pl == 1 ? (const void*)a.xv : pl == 2 ? (const void*)a.o.Na
                        : pl == 3 ? (const void*)a.o.Nb : pl == 4 ? (const void*)a.o.Bx : pl == 5 ? (const void*)a.o.By
                        : pl == 6 ? (const void*)a.idu : pl == 7 ? (const void*)a.idv
                        : pl == 8 ? (const void*)a.bu : (const void*)a.bv;
    const char* src = static_cast<const char*>(plane) + ((long long)(i0 + hc) * d.ld + j0 + r0) * (long long)es;
    const uint32_t pitch = 2 * d.ld * es;
    const uint32_t dcol = (pl < 8 ? COL : 2 * RP) * es;
    const uint32_t dst0 = (pl < 8 ? smem_addr(ring + pl * RP + r0) : smem_addr(bring + (pl - 8) * RP + r0)) + hc * dcol;
    const uint32_t cbytes = cr1 > cr0 ? (cr1 - cr0) * sizeof(double) : 0;
    const uint32_t bar0 = smem_addr(&bars[0]);
    const int npair = tw / 2 + H + (tw & 1);   // pairs of the region (an odd width's last column is beyond it)
    int slot = 0;
    // A wait that runs out fails the solve: the lane issues nothing more, so that soon the waits of all
    // run out, and the block goes on over what there is, its barriers unchanged.
    bool ok = !a.drop;
    auto coarse_total = [&](int C) {
      return ((coarse_col(a.oc, C, true) >= 0 ? 1u : 0u) + (coarse_col(a.oc, C, false) >= 0 ? 1u : 0u)) * cbytes;
    };
    auto issue = [&](int t) {
      const int i = i0 + 2 * t;
      const uint32_t bar = bar0 + (t & (kWaveBars - 1)) * 8;
      if (mover) {
        const bool in0 = i >= 0 && i < d.nx, in1 = i + 1 >= 0 && i + 1 < d.nx;
        if (lane == 0 && ok) {
          // x has been written by other threads since its last copy
          if (UP && w == 0) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                       "r"((in0 ? sum[0] : 0u) + (in1 ? sum[1] : 0u))
                       : "memory");
        }
        __syncwarp();
        if (bytes && ok && (hc ? in1 : in0)) bulk_copy(dst0 + slot * dcol, src, bytes, bar);
      } else if (UP) {
        // coarse columns that arrive with the pair: fx = 2, the one beyond that of its even column
        // (with the first pair also those before it); fx = 1, the pair's own
        const int Cb = a.fx == 1 ? i + 1 : ((i + 1) >> 1) + 1, Ca = a.fx == 1 ? i : t == 0 ? Cb - 3 : Cb;
        if (lane == 0 && ok) {
          uint32_t total = 0;
          for (int C = Ca; C <= Cb; ++C) total += coarse_total(C);
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(total) : "memory");
        }
        __syncwarp();
        if (lane < 2 && cbytes && ok)
          for (int C = Ca; C <= Cb; ++C) {
            const int I = coarse_col(a.oc, C, lane == 0);
            if (I >= 0)
              bulk_copy(smem_addr(cring + ((C & (kWaveCoarse - 1)) * 2 + lane) * CP + cr0),
                        (lane == 0 ? a.xcu : a.xcv) + (long long)I * a.oc.d.ld + CJ0 + cr0, cbytes, bar);
          }
      } else {   // the descent enters a level with x = 0
        constexpr int n16 = 2 * RP * sizeof(double) / 16;
        for (int t2 = lane; t2 < 2 * n16; t2 += 32)
          reinterpret_cast<uint4*>(ring + (slot + t2 / n16) * COL)[t2 % n16] = make_uint4(0u, 0u, 0u, 0u);
        if (lane == 0 && ok)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
      }
      src += pitch;
      slot = slot == NC - 2 ? 0 : slot + 2;
    };
    auto arrived = [&](int t) { return wave_wait(bar0 + (t & (kWaveBars - 1)) * 8, (t / kWaveBars) & 1); };
    int next = 0, waited = 0, issued = npair;   // the pair to issue, those that have arrived, those a lane issued
    auto wait_next = [&] {
      ok = arrived(waited);
      if (ok) ++waited;
      else issued = a.drop ? 0 : next;
    };
    while (next < kWavePre && next < npair) issue(next++);
    wait_next();
    if (ok) wait_next();
    __syncthreads();
#pragma unroll 1
    for (int s = 0; s <= last; ++s) {
      if (next < npair) issue(next++);
      if (ok && waited < npair) wait_next();   // the next step reads up to pair s + 2
      __syncthreads();
    }
    for (; waited < issued; ++waited) ok = arrived(waited) && ok;   // no copy in flight when the block ends
    if (!ok) *a.fail = 1.0;
  } else {
    // ---- x += P x_c (prolong_delta's taps, weights and order)
    const int t0 = (warp - NPW - NOUT - kWaveCopy) * 32 + lane, r = t0 % RP, comp = (t0 / RP) & 1, h = t0 / (2 * RP);
    const int j = j0 + r;
    const Dims& dc = a.oc.d;
    const int il = comp == 0 ? d.nx - 3 : d.nx - 2, jl = comp == 0 ? d.ny - 2 : d.ny - 3;
    const int lj = comp == 0 ? dc.ny - 1 : dc.ny - 2, li = comp == 0 ? dc.nx - 2 : dc.nx - 1;   // coarse: last row, column
    const int gW = comp == 0 ? bc.uW : bc.vW, gE = comp == 0 ? bc.uE : bc.vE;
    const int gS = comp == 0 ? bc.uS : bc.vS, gN = comp == 0 ? bc.uN : bc.vN;
    const bool row = r < RP - 1 && j >= 1 && j <= jl;   // (the ring's last row is no halo row)
    int Cj[2];
    double wj[2];
    two_taps(j, a.fy, comp == 1, Cj, wj);
    // the taps' coarse rows, clamped and through the boundary rule of an interior column (-1: zero)
    const int cS = comp == 0 ? a.oc.bc.uS : a.oc.bc.vS, cN = comp == 0 ? a.oc.bc.uN : a.oc.bc.vN;
    int J[2], Jr[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      J[e] = min(max(Cj[e], 0), lj);
      Jr[e] = J[e] == 0 ? (cS == kINF ? 1 : -1) : J[e] == lj ? (cN == kINF ? lj - 1 : -1) : J[e];
    }
    const double* cp = cring + comp * CP;
    double* x = ring + comp * RP;
    const int c0 = 1 - i0, c1 = min(ncols - 1, il - i0);
    int cc = 0, off = 0;
    __syncthreads();
#pragma unroll 1
    for (int s = 0; s <= last; ++s, cc += 2, off = next2(off)) {
      const int c = cc + h, o = off + h * COL;   // (a pair's slots are neighbours)
      if (row && c >= c0 && c <= c1) {
        const int i = i0 + c;
        int Ci[2];
        double wi[2];
        two_taps(i, a.fx, comp == 0, Ci, wi);
        const int I0 = min(max(Ci[0], 0), li), I1 = min(max(Ci[1], 0), li);
        double v[2][2];
        const bool iedge = I0 == 0 || I0 == li || I1 == 0 || I1 == li;
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int f = 0; f < 2; ++f) {
            int jr = Jr[e], js, is;
            if (iedge)   // the corners' rule (the column is mapped already)
              jr = (comp == 0 ? u_src(dc, a.oc.bc, J[e], f ? I1 : I0, js, is)
                              : v_src(dc, a.oc.bc, J[e], f ? I1 : I0, js, is)) ? js : -1;
            v[e][f] = jr >= 0 ? cp[(Ci[f] & (kWaveCoarse - 1)) * 2 * CP + jr - CJ0] : 0.0;
          }
        double t = (wj[0] * wi[0]) * v[0][0];
        t = fma(wj[0] * wi[1], v[0][1], t);
        t = fma(wj[1] * wi[0], v[1][0], t);
        t = fma(wj[1] * wi[1], v[1][1], t);
        const RIx ix = beside(o, i);
        const double val = x[o + r] + t;
        x[o + r] = val;
        if (j == 1 || j == jl || i == 1 || i == il) ghosts(x, ix, j, i, il, jl, gW, gE, gS, gN, val);
      }
      __syncthreads();
    }
  }
}

// the restricted residual of the finer level as this level's right-hand side
__global__ void k_restrict_b(Dims df, Dims dc, int fx, int fy, const double* ru, const double* rv, double* bu, double* bv) {
  IDX2D
  if (j >= dc.ny || i >= dc.nx) return;
  const long long q = dc.at(j, i);
  double b0, b1;
  restrict_values(df, dc, fx, fy, ru, rv, j, i, b0, b1);
  bu[q] = b0;
  bv[q] = b1;
}

// ---- direct solve of the coarsest level ------------------------------------------------
// The coarsest level has at most kCoarseDirectMax interior unknowns, numbered u first,
// then v, each in plane order (i outer, j inner).  Once per viscosity iteration its
// reduced matrix is assembled from the sub-cycle's row tables (the operator's nine
// terms per row, boundary reads already mapped to their sources, duplicates summed in
// the operator's own term order) and inverted by Gauss-Jordan elimination with partial
// pivoting, in one launch; the coarse step of every V-cycle is then one matrix-vector
// product.  A pivot below 1e-13 of the largest entry (a singular coarse operator, e.g.
// a free-floating shelf with no fixed boundary) raises the flag and the coarse step
// relaxes instead.
struct CoarseMap {
  int ny, nu, nv;
  __host__ __device__ __forceinline__ int n() const { return nu + nv; }
};

// Assembly and inversion of the coarsest level's matrix by the first threads of a block.  tab is the
// level's row table (of R = n rows: 4 same-component and 4 cross-component mapped reads of each,
// then their own positions; the zero element P = nx*ny stands for 'zero' sides); o reads
// compact planes (row length ny).  Gauss-Jordan step k maps the matrix of step k-1 (buffer k&1)
// to the next one in one pass with one barrier: every warp finds the pivot row p of column k
// itself, and every element takes its value from the old matrix with rows k and p exchanged.
// Bound by the latency of the n steps (pivot search, division, barrier): eight warps, a lane to a
// column (two at most), so that a step takes one division per column and warp and the
// redundant search stays cheap (a step takes 1100 cycles at n = 12, 1500 at 31; a thread per
// element was no faster).
constexpr int kInvThreads = 1024;   // of the set-up kernel
constexpr int kInvWarps = 8;
constexpr size_t kInvDbl = 2 * kCoarseDirectMax * (kCoarseDirectMax + 1);

__device__ __forceinline__ void coarse_setup_block(const Op& o, const CoarseMap& m, const uint16_t* tab,
                                                   double* inv_buf, double* Ainv, int* singular) {
  constexpr int M = kCoarseDirectMax, LD = M + 1;
  __shared__ int perm[M];
  __shared__ double wmax[kInvWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = m.n(), ny = m.ny, P = o.d.nx * ny;
  constexpr int threads = 32 * kInvWarps;
  if (tid >= threads) return;
  auto barrier = [&] {
    __syncwarp();
    asm volatile("bar.sync 1, %0;" ::"n"(threads) : "memory");
  };
  const Dims& d = o.d;
  for (int e = tid; e < n * n; e += threads) inv_buf[(e / n) * LD + e % n] = 0.0;
  barrier();
  // the unknown of a plane position (compact rows of length ny) of a u or v point
  auto unknown = [&](int pos, bool ucomp) {
    const int i = pos / ny, j = pos % ny;
    return ucomp ? (i - 1) * (ny - 2) + (j - 1) : m.nu + (i - 1) * (ny - 3) + (j - 1);
  };
  for (int r = tid; r < n; r += threads) {
    const int pos = tab[8 * n + r], i = pos / ny, j = pos % ny;   // (tab_pos)
    int src[8];
    for (int t = 0; t < 8; ++t) src[t] = tab[8 * r + t];
    double cf[9];
    if (r < m.nu) {
      const double Ae = o.Na[d.at(j, i + 1)], Aw = o.Na[d.at(j, i)], Bn = o.Nb[d.at(j, i)], Bs = o.Nb[d.at(j - 1, i)];
      const double cE = 4.0 * o.ax * Ae, cW = 4.0 * o.ax * Aw, cN = o.ay * Bn, cS = o.ay * Bs;
      cf[0] = cE; cf[1] = cW; cf[2] = cN; cf[3] = cS;
      cf[4] = -(cE + cW + cN + cS) - o.Bx[d.at(j, i)];
      cf[5] = -2.0 * Aw - Bn; cf[6] = 2.0 * Ae + Bn; cf[7] = 2.0 * Aw + Bs; cf[8] = -2.0 * Ae - Bs;
    } else {
      const double An = o.Na[d.at(j + 1, i)], As = o.Na[d.at(j, i)], Be = o.Nb[d.at(j, i)], Bw = o.Nb[d.at(j, i - 1)];
      const double cN = 4.0 * o.ay * An, cS = 4.0 * o.ay * As, cE = o.ax * Be, cW = o.ax * Bw;
      cf[0] = cN; cf[1] = cS; cf[2] = cE; cf[3] = cW;
      cf[4] = -(cN + cS + cE + cW) - o.By[d.at(j, i)];
      cf[5] = -2.0 * An - Bw; cf[6] = 2.0 * An + Be; cf[7] = 2.0 * As + Bw; cf[8] = -2.0 * As - Be;
    }
    const bool u = r < m.nu;
    const int row = unknown(pos, u);
    double* a = inv_buf + row * LD;
    // the terms in the operator's order: 4 same-component reads, the diagonal, 4 cross reads
    for (int t = 0; t < 4; ++t)
      if (src[t] != P) a[unknown(src[t], u)] += cf[t];
    a[row] += cf[4];
    for (int t = 4; t < 8; ++t)
      if (src[t] != P) a[unknown(src[t], !u)] += cf[t + 1];
  }
  barrier();
  double amax = 0.0;
  for (int e = tid; e < n * n; e += threads) {
    const double v = inv_buf[(e / n) * LD + e % n];
    amax = (fabs(v) > amax || v != v) ? fabs(v) : amax;
  }
  for (int o2 = 16; o2 > 0; o2 >>= 1) {   // largest magnitude; a NaN wins
    const double w = __shfl_xor_sync(0xffffffffu, amax, o2);
    amax = (w > amax || w != w) ? w : amax;
  }
  if (lane == 0) wmax[warp] = amax;
  barrier();
  amax = wmax[0];
  for (int w = 1; w < kInvWarps; ++w) amax = (wmax[w] > amax || wmax[w] != wmax[w]) ? wmax[w] : amax;
  const double tiny = 1e-13 * amax;
  bool bad = !(amax > 0.0) || amax != amax;
  static_assert(M <= 64, "two columns per lane");
  int cur = 0;
  for (int k = 0; k < n && !bad; ++k) {
    const double* a = inv_buf + cur * M * LD;
    double* b = inv_buf + (cur ^ 1) * M * LD;
    // pivot: largest |a[r][k]|, r >= k, lowest r on ties (the same in every warp; magnitudes
    // compare like their bits, a NaN counts as zero)
    int br = k + lane;
    double best = br < n ? fabs(a[br * LD + k]) : 0.0;
    const double second = br + 32 < n ? fabs(a[(br + 32) * LD + k]) : 0.0;
    if (best != best) best = 0.0;
    if (second > best) { best = second; br += 32; }
    const unsigned hi = (unsigned)__double2hiint(best), top = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = hi == top ? (unsigned)__double2loint(best) : 0u, low = __reduce_max_sync(0xffffffffu, lo);
    const bool wins = br < n && hi == top && (unsigned)__double2loint(best) == low;
    const int p = __reduce_min_sync(0xffffffffu, wins ? br : n);
    if (!(__hiloint2double((int)top, (int)low) > tiny)) { bad = true; break; }
    if (tid == 0) perm[k] = p;
    const double piv = a[p * LD + k];
    double pk[2];   // the normalised pivot row at this lane's columns
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = lane + 32 * h;
      if (c >= n) continue;
      pk[h] = (c == k ? 1.0 : a[p * LD + c]) / piv;
    }
    for (int r = warp; r < n; r += kInvWarps) {
      const int src = r == p ? k : r;   // the row that sits at r after the exchange
      const double f = a[src * LD + k];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = lane + 32 * h;
        if (c < n) b[r * LD + c] = r == k ? pk[h] : (c == k ? 0.0 : a[src * LD + c]) - f * pk[h];
      }
    }
    cur ^= 1;
    barrier();
  }
  if (!bad) {   // columns back in order: the row exchanges undone from the last to the first
    const double* a = inv_buf + cur * M * LD;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = lane + 32 * h;
      if (c >= n) continue;
      int from = c;
      for (int k = 0; k < n; ++k) from = from == k ? perm[k] : (from == perm[k] ? k : from);
      for (int r = warp; r < n; r += kInvWarps) Ainv[r * n + c] = a[r * LD + from];
    }
  }
  if (tid == 0) *singular = bad ? 1 : 0;
}


// The levels from `first` down, run by one thread block out of shared memory with barriers
// between the phases (colour passes, residual, transfers), without a launch and a global-memory
// round trip per phase.  Each level keeps kSubArrays compact planes (row length ny, one extra
// element that stays 0) in the block's dynamic shared memory; the coefficients of every level
// are copied in at the start, x of the first level is written back at the end.
//
// Bound by the latency of a phase, not by its points (a coarse level has a handful), so a phase
// keeps only what depends on the phase before it.  The interior rows of a level are grouped by
// (component, colour); a quarter of the block (kSubQuarter threads) belongs to each of the four
// groups.  On the levels of at most kSubQuarter rows a group a thread has one row ("resident"):
// it loads the row's coefficients, its neighbours' addresses and b when it comes to the level,
// ahead of the passes that need them, and a pass is nine reads of x, three chains of three
// multiply-adds and a write; the levels' phases are separated by named barriers of the threads
// that have rows there, while the others wait at the level above.  Larger levels load a row's
// operands in the pass, every thread on every class.  (With every thread at every barrier and
// all operands loaded in every pass, a pass over three rows a group took 650 cycles, now 400;
// the kernel 27.3 -> 22.7 us from 65 x 9 points, 30 -> 24.7 us from 40 x 23.  Launching the next
// kernel ahead of the end of the last saved 0.2 us a launch in a graph, not worth its waits.)
//
// The row tables are built once on the host (they depend on the grid and the boundary
// conditions only), per level of R rows: the positions of each row's eight off-diagonal reads
// (boundary unknowns resolved to their sources, 'zero' sides to the zero element), its own
// position, its prolongation taps from the next level and, below the first level, its
// restriction taps from the level above, each a position and a weight in sixteenths.
enum { SA_NA, SA_NB, SA_BX, SA_BY, SA_IDU, SA_IDV, SA_XU, SA_XV, SA_BU, SA_BV, kSubArrays };
constexpr size_t kSubSmemBudget = 200 * 1024;   // of a level and those below it (sub_bytes)
constexpr size_t kSubSmemMax = 224 * 1024;      // with the restriction taps and the residual
constexpr int kSubQuarter = kSubThreads / 4;
constexpr int kTabReads = 8, kTabProlong = 4, kTabRestrict = 12;   // entries per row
constexpr int kTapBits = 12;   // a tap: position, and above it 16 x weight - 1
// where a level's blocks of the table start: reads, positions (padded to 4), prolongation, restriction
__host__ __device__ __forceinline__ int tab_pos(int R) { return kTabReads * R; }
__host__ __device__ __forceinline__ int tab_prolong(int R) { return tab_pos(R) + (R + 3) / 4 * 4; }
__host__ __device__ __forceinline__ int tab_restrict(int R) { return tab_prolong(R) + kTabProlong * R; }

struct SubLevel {
  Op o;                      // global-memory operator of the level
  const double *idu, *idv;   // global inverse diagonals
  int soff;                  // offset of the level's planes in shared memory (doubles)
  int rows;                  // interior rows (u then v)
  int cls[5];                // row ranges of the classes u colour 0, u 1, v 0, v 1
  int most;                  // rows of the largest class
  int toff;                  // offset of the level's row table in the shared table area (uint16)
  const uint16_t* gtab;      // the table in global memory
};
struct SubCycle {
  int first, last, nu1, nu2, coarse_sweeps;
  int direct;                  // coarsest level solved with Ainv unless *singular
  CoarseMap map;
  const double* Ainv;
  const int* singular;
  Restriction rs;              // b of the first level: given, or restricted from the finer residual
  int dbl;                     // doubles of all levels' planes (the table area follows)
  int ainv_off;                // offset (doubles) of the staged inverse, after the tables
  int res_off;                 // the residual of the level being left: u, v (a zero element before each)
  int tab16;                   // 16-byte vectors of all levels' row tables
  SubLevel L[kMaxLevels];
};

__device__ __forceinline__ void copy8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ double lds(uint32_t at) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(at));
  return v;
}
__device__ __forceinline__ void sts(uint32_t at, double v) { asm volatile("st.shared.f64 [%0], %1;" ::"r"(at), "d"(v)); }

// A level of the sub-cycle in shared memory: its planes, its row table and the operator's scale.
struct SubMem {
  double* a;
  const uint16_t* tab;
  int P1, ny, R;
  double ax, ay;
  __device__ __forceinline__ SubMem(const SubCycle& sc, double* sm, const uint16_t* tabs, int l) {
    const SubLevel& L = sc.L[l];
    a = sm + L.soff;
    tab = tabs + L.toff;
    ny = L.o.d.ny;
    P1 = L.o.d.nx * ny + 1;
    R = L.rows;
    ax = L.o.ax;
    ay = L.o.ay;
  }
  __device__ __forceinline__ double* plane(int k) const { return a + k * P1; }
  __device__ __forceinline__ int pos(int r) const { return tab[tab_pos(R) + r]; }
};
// N_a and N_b a row takes, in the order A1 A0 B1 B0 of row_terms, and its diagonal
template <bool U>
__device__ __forceinline__ void row_coefficients(const SubMem& m, int q, double (&c)[5]) {
  const double *Na = m.plane(SA_NA), *Nb = m.plane(SA_NB), pa = U ? m.ax : m.ay, pb = U ? m.ay : m.ax;
  c[0] = U ? Na[q + m.ny] : Na[q + 1];
  c[1] = Na[q];
  c[2] = Nb[q];
  c[3] = U ? Nb[q - 1] : Nb[q - m.ny];
  c[4] = -(4.0 * pa * c[0] + 4.0 * pa * c[1] + pb * c[2] + pb * c[3]) - m.plane(U ? SA_BX : SA_BY)[q];
}
// (A x) of a u (v) row: the operator's nine terms (AuXC, AvXC) in three chains.  x: the row's own
// value, then its four neighbours of the same component and the four of the other.
template <bool U>
__device__ __forceinline__ double row_terms(const double (&c)[5], double ax, double ay, const double (&x)[9]) {
  const double A1 = c[0], A0 = c[1], B1 = c[2], B0 = c[3], pa = U ? ax : ay, pb = U ? ay : ax;
  double s0 = 4.0 * pa * A1 * x[1], s1 = 4.0 * pa * A0 * x[2], s2 = pb * B1 * x[3];
  s0 = fma(pb * B0, x[4], s0);
  s1 = fma(c[4], x[0], s1);
  s2 = fma(U ? -2.0 * A0 - B1 : -2.0 * A1 - B0, x[5], s2);
  s0 = fma(2.0 * A1 + B1, x[6], s0);
  s1 = fma(2.0 * A0 + B0, x[7], s1);
  s2 = fma(U ? -2.0 * A1 - B0 : -2.0 * A0 - B1, x[8], s2);
  return (s0 + s1) + s2;
}
// the same from the tables (x, y: the planes of the row's component and of the other)
template <bool U>
__device__ __forceinline__ double row_apply(const SubMem& m, int r, int& q, const double* x, const double* y) {
  const uint4 at = reinterpret_cast<const uint4*>(m.tab)[r];
  q = m.pos(r);
  double c[5];
  row_coefficients<U>(m, q, c);
  const double v[9] = {x[q], x[at.x & 0xffffu], x[at.x >> 16], x[at.y & 0xffffu], x[at.y >> 16],
                       y[at.z & 0xffffu], y[at.z >> 16], y[at.w & 0xffffu], y[at.w >> 16]};
  return row_terms<U>(c, m.ax, m.ay, v);
}

__global__ void __launch_bounds__(kSubThreads) k_subcycle(const __grid_constant__ SubCycle sc, double* xu0,
                                                          double* xv0, const double* bu0, const double* bv0) {
  extern __shared__ double sm[];
  __shared__ double weight[16], sr[kCoarseDirectMax];
  __shared__ uint16_t number[kCoarseDirectMax], place[kCoarseDirectMax];   // unknown of a coarsest row; its position
  uint16_t* tabs = reinterpret_cast<uint16_t*>(sm + sc.dbl);
  double* Ainv = sm + sc.ainv_off;
  const int tid = threadIdx.x, quarter = tid / kSubQuarter, t = tid % kSubQuarter;
  const bool urow = quarter < 2;   // (of a resident row)
  // whether the coarsest level is solved with its inverse (the flag's load overlaps the copies)
  const bool direct = sc.direct && *sc.singular == 0;
  if (tid < 16) weight[tid] = 0.0625 * (tid + 1);
  {
    int total = 0;
    for (int l = sc.first; l <= sc.last; ++l) total += sc.L[l].o.d.nx * sc.L[l].o.d.ny + 1;
    for (int t0 = tid; t0 < total; t0 += kSubThreads) {
      int l = sc.first, e = t0;
      while (e >= sc.L[l].o.d.nx * sc.L[l].o.d.ny + 1) { e -= sc.L[l].o.d.nx * sc.L[l].o.d.ny + 1; ++l; }
      const SubLevel& L = sc.L[l];
      const Dims& d = L.o.d;
      const int P = d.nx * d.ny, P1 = P + 1;
      double* a = sm + L.soff;
      a[SA_XU * P1 + e] = 0.0;   // every level is entered with x = 0
      a[SA_XV * P1 + e] = 0.0;
      if (e == P) continue;
      const long long q = d.at(e % d.ny, e / d.ny);
      copy8(a + SA_NA * P1 + e, L.o.Na + q);
      copy8(a + SA_NB * P1 + e, L.o.Nb + q);
      copy8(a + SA_BX * P1 + e, L.o.Bx + q);
      copy8(a + SA_BY * P1 + e, L.o.By + q);
      copy8(a + SA_IDU * P1 + e, L.idu + q);
      copy8(a + SA_IDV * P1 + e, L.idv + q);
    }
    // the levels' tables are contiguous and padded to 16 bytes in both places
    const uint4* g = reinterpret_cast<const uint4*>(sc.L[sc.first].gtab);
    for (int e = tid; e < sc.tab16; e += kSubThreads) copy16(reinterpret_cast<uint4*>(tabs) + e, g + e);
    if (direct)
      for (int e = tid, n = sc.map.n(); e < n * n; e += kSubThreads) copy8(Ainv + e, sc.Ainv + e);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (direct && tid >= kSubThreads - kCoarseDirectMax && tid - (kSubThreads - kCoarseDirectMax) < sc.map.n()) {
      const SubLevel& L = sc.L[sc.last];
      const int r = tid - (kSubThreads - kCoarseDirectMax), ny = sc.map.ny, q = L.gtab[tab_pos(L.rows) + r];
      const int i = q / ny, j = q % ny, k = r < L.cls[2] ? (i - 1) * (ny - 2) + j - 1 : sc.map.nu + (i - 1) * (ny - 3) + j - 1;
      number[r] = (uint16_t)k;
      place[k] = (uint16_t)q;
    }
    const SubLevel& L = sc.L[sc.first];
    const Dims& d = L.o.d;
    const int P = d.nx * d.ny, P1 = P + 1;
    double* a = sm + L.soff;
    for (int e = tid; e < P; e += kSubThreads) {
      const int j = e % d.ny, i = e / d.ny;
      double b0, b1;
      if (sc.rs.on) {
        restrict_from(sc.rs, d, j, i, b0, b1);
      } else {
        const long long q = d.at(j, i);
        b0 = bu0[q];
        b1 = bv0[q];
      }
      a[SA_BU * P1 + e] = b0;
      a[SA_BV * P1 + e] = b1;
    }
    if (tid == 0) sm[sc.res_off] = sm[sc.res_off + P1] = 0.0;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
  __syncthreads();
  double* ru = sm + sc.res_off + 1;
  double* rv = ru + sc.L[sc.first].o.d.nx * sc.L[sc.first].o.d.ny + 1;
  auto tap = [&](const double* x, uint32_t e, double s) {
    return fma(weight[e >> kTapBits], x[e & ((1u << kTapBits) - 1)], s);
  };
  // b of a row from the residual of the level above (restrict_values' taps and order)
  auto restricted = [&](const SubMem& m, int r, bool u) {
    const uint2* e = reinterpret_cast<const uint2*>(m.tab + tab_restrict(m.R)) + 3 * r;
    const double* f = (u ? ru : rv) - 1;
    const uint2 v0 = e[0], v1 = e[1], v2 = e[2];
    double s = tap(f, v0.x & 0xffffu, 0.0);
    s = tap(f, v0.x >> 16, s); s = tap(f, v0.y & 0xffffu, s); s = tap(f, v0.y >> 16, s);
    s = tap(f, v1.x & 0xffffu, s); s = tap(f, v1.x >> 16, s); s = tap(f, v1.y & 0xffffu, s); s = tap(f, v1.y >> 16, s);
    s = tap(f, v2.x & 0xffffu, s); s = tap(f, v2.x >> 16, s); s = tap(f, v2.y & 0xffffu, s); s = tap(f, v2.y >> 16, s);
    return s;
  };
  // (P x_c) of a row (prolong_delta's taps and order)
  auto prolonged = [&](const SubMem& m, const SubMem& k, int r, bool u) {
    const uint2 e = reinterpret_cast<const uint2*>(m.tab + tab_prolong(m.R))[r];
    const double* f = k.plane(u ? SA_XU : SA_XV);
    double s = tap(f, e.x & 0xffffu, 0.0);
    s = tap(f, e.x >> 16, s);
    s = tap(f, e.y & 0xffffu, s);
    return tap(f, e.y >> 16, s);
  };
  // ---- the levels with more rows than the block has threads for them: every thread on every row
  auto gs_pass = [&](const SubMem& m, int l, int p) {
    double *xu = m.plane(SA_XU), *xv = m.plane(SA_XV);
    for (int r = sc.L[l].cls[p] + tid; r < sc.L[l].cls[p + 1]; r += kSubThreads) {
      int q;
      if (p < 2) {
        const double Ax = row_apply<true>(m, r, q, xu, xv);
        xu[q] = fma(m.plane(SA_BU)[q] - Ax, m.plane(SA_IDU)[q], xu[q]);
      } else {
        const double Ax = row_apply<false>(m, r, q, xv, xu);
        xv[q] = fma(m.plane(SA_BV)[q] - Ax, m.plane(SA_IDV)[q], xv[q]);
      }
    }
    __syncthreads();
  };
  int tail = sc.first;   // the first level of resident rows; none where the coarsest level is relaxed
  while (direct ? sc.L[tail].most > kSubQuarter : tail <= sc.last) ++tail;
  for (int l = sc.first; l < tail; ++l) {
    const SubMem m(sc, sm, tabs, l);
    double *xu = m.plane(SA_XU), *xv = m.plane(SA_XV);
    if (l > sc.first) {
      for (int r = tid; r < m.R; r += kSubThreads) {
        const bool u = r < sc.L[l].cls[2];
        m.plane(u ? SA_BU : SA_BV)[m.pos(r)] = restricted(m, r, u);
      }
      __syncthreads();
    }
    if (l == sc.last) {   // relaxed: symmetric sweeps u0 u1 v0 v1 | v1 v0 u1 u0
      for (int s = 0; s < 8 * sc.coarse_sweeps; ++s) gs_pass(m, l, s & 4 ? 3 - (s & 3) : s & 3);
      break;
    }
    for (int s = 0; s < 4 * sc.nu1; ++s) gs_pass(m, l, s & 3);
    // residual of the interior rows (the restriction reads interior rows only)
    for (int r = tid; r < m.R; r += kSubThreads) {
      int q;
      if (r < sc.L[l].cls[2]) {
        const double Ax = row_apply<true>(m, r, q, xu, xv);
        ru[q] = m.plane(SA_BU)[q] - Ax;
      } else {
        const double Ax = row_apply<false>(m, r, q, xv, xu);
        rv[q] = m.plane(SA_BV)[q] - Ax;
      }
    }
    __syncthreads();
  }
  // ---- the levels of resident rows: a quarter's first `width` threads (whole warps) have the
  // rows of its class (`most` does not grow from a level to the next)
  auto width_of = [&](int l) { return max(1, (sc.L[l].most + 31) / 32) * 32; };
  if (tail <= sc.last && t < width_of(tail)) {
    int l = tail;
    bool up = false;
    while (true) {
      const SubMem m(sc, sm, tabs, l);
      const int width = width_of(l), bar = 1 + l - tail;
      auto barrier = [&] {   // of the level's threads
        __syncwarp();
        asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(4 * width) : "memory");
      };
      if (!up && l == sc.last) {   // x = Ainv b, eight threads to a row
        const int flat = quarter * width + t, n = sc.map.n();
        for (int r = flat; r < m.R; r += 4 * width) {
          const bool u = r < sc.L[l].cls[2];
          sr[number[r]] = l > sc.first ? restricted(m, r, u) : m.plane(u ? SA_BU : SA_BV)[m.pos(r)];
        }
        barrier();
        for (int r0 = 0; r0 < n; r0 += width / 2) {
          const int r = r0 + flat / 8;
          double s = 0.0;
          if (r < n)
            for (int c = flat % 8; c < n; c += 8) s += Ainv[r * n + c] * sr[c];
          s += __shfl_xor_sync(0xffffffffu, s, 4);
          s += __shfl_xor_sync(0xffffffffu, s, 2);
          s += __shfl_xor_sync(0xffffffffu, s, 1);
          if (r < n && flat % 8 == 0) m.plane(r < sc.map.nu ? SA_XU : SA_XV)[place[r]] = s;
        }
        if (l == tail) break;
        up = true;
        --l;
        continue;
      }
      const int r = sc.L[l].cls[quarter] + t;
      const bool on = r < sc.L[l].cls[quarter + 1];
      // the row's neighbours (shared-memory addresses), coefficients, inverse diagonal and b
      uint32_t at[9], atb = 0;
      double c[5] = {}, id = 0.0, b = 0.0;
      int q = 0;
      if (on) {
        const uint4 e = reinterpret_cast<const uint4*>(m.tab)[r];
        const uint32_t x = smem_addr(m.plane(urow ? SA_XU : SA_XV)), y = smem_addr(m.plane(urow ? SA_XV : SA_XU));
        q = m.pos(r);
        at[0] = x + 8 * q;
        at[1] = x + 8 * (e.x & 0xffffu); at[2] = x + 8 * (e.x >> 16);
        at[3] = x + 8 * (e.y & 0xffffu); at[4] = x + 8 * (e.y >> 16);
        at[5] = y + 8 * (e.z & 0xffffu); at[6] = y + 8 * (e.z >> 16);
        at[7] = y + 8 * (e.w & 0xffffu); at[8] = y + 8 * (e.w >> 16);
        atb = smem_addr(m.plane(urow ? SA_BU : SA_BV) + q);
        if (urow) row_coefficients<true>(m, q, c);
        else row_coefficients<false>(m, q, c);
        id = m.plane(urow ? SA_IDU : SA_IDV)[q];
      }
      if (up) {   // x += P x_c, once the level below is done
        barrier();
        if (on) sts(at[0], lds(at[0]) + prolonged(m, SubMem(sc, sm, tabs, l + 1), r, urow));
        barrier();
      } else if (l > sc.first && on) {
        sts(atb, restricted(m, r, urow));
      }
      if (on) b = lds(atb);
      auto rest = [&] {   // b - A x of the row; its x
        double v[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) v[k] = lds(at[k]);
        const double Ax = urow ? row_terms<true>(c, m.ax, m.ay, v) : row_terms<false>(c, m.ax, m.ay, v);
        return make_double2(b - Ax, v[0]);
      };
      for (int s = 4 * (up ? sc.nu2 : sc.nu1); s > 0; --s) {   // in the ascent the other way round
        if (on && quarter == (up ? (s - 1) & 3 : -s & 3)) {
          const double2 f = rest();
          sts(at[0], fma(f.x, id, f.y));
        }
        barrier();
      }
      if (up) {
        if (l == tail) break;
        --l;
        continue;
      }
      if (on) (urow ? ru : rv)[q] = rest().x;
      barrier();
      if (t < width_of(l + 1)) ++l;
      else up = true;   // no rows below: on to this level's ascent
    }
  }
  __syncthreads();
  for (int l = min(tail, sc.last) - 1; l >= sc.first; --l) {
    const SubMem m(sc, sm, tabs, l), k(sc, sm, tabs, l + 1);
    for (int r = tid; r < m.R; r += kSubThreads) {
      const bool u = r < sc.L[l].cls[2];
      m.plane(u ? SA_XU : SA_XV)[m.pos(r)] += prolonged(m, k, r, u);
    }
    __syncthreads();
    for (int s = 4 * sc.nu2 - 1; s >= 0; --s) gs_pass(m, l, s & 3);
  }
  {
    const SubMem m(sc, sm, tabs, sc.first);
    const double *xu = m.plane(SA_XU), *xv = m.plane(SA_XV);
    for (int e = tid; e < m.P1 - 1; e += kSubThreads) {
      const long long q = sc.L[sc.first].o.d.at(e % m.ny, e / m.ny);
      xu0[q] = xu[e];
      xv0[q] = xv[e];
    }
  }
}

// rediscretised coarse coefficients (averages of the fine ones; B scales with the cell area)
__device__ __forceinline__ int clamp_index(int v, int hi) { return v < 0 ? 0 : (v > hi ? hi : v); }
// weights of the full weighting, offsets -1, 0, 1 (the middle alone in a direction not coarsened)
__device__ __forceinline__ double full_weight(int a, int f) { return f == 2 ? (a == 0 ? 0.5 : 0.25) : (a == 0 ? 1.0 : 0.0); }
__device__ __forceinline__ double coarsen_Na(const Dims& df, int fx, int fy, const double* Na, int j, int i) {
  double s = 0.0;   // around fine a (fy*j, fx*i)
#pragma unroll
  for (int a = -1; a <= 1; ++a)
#pragma unroll
    for (int b = -1; b <= 1; ++b) {
      const double w = full_weight(a, fy) * full_weight(b, fx);
      if (w != 0.0) s += w * Na[df.at(clamp_index(fy * j + a, df.ny - 1), clamp_index(fx * i + b, df.nx - 1))];
    }
  return s;
}
__device__ __forceinline__ double coarsen_Nb(const Dims& df, int fx, int fy, const double* Nb, int j, int i) {
  double s = 0.0;   // fine b cells inside the coarse b cell
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b)
      if (a < fy && b < fx) s += Nb[df.at(clamp_index(fy * j + a, df.ny - 2), clamp_index(fx * i + b, df.nx - 2))];
  return s / (double)(fy * fx);
}
__device__ __forceinline__ double coarsen_Bx(const Dims& df, int fx, int fy, const double* Bx, int j, int i) {
  double s = 0.0;   // cell along x, node along y
#pragma unroll
  for (int a = -1; a <= 1; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const double w = full_weight(a, fy) * (1.0 / fx);
      if (w != 0.0 && b < fx) s += w * Bx[df.at(clamp_index(fy * j + a, df.ny - 1), clamp_index(fx * i + b, df.nx - 2))];
    }
  return (double)(fx * fy) * s;
}
__device__ __forceinline__ double coarsen_By(const Dims& df, int fx, int fy, const double* By, int j, int i) {
  double s = 0.0;   // cell along y, node along x
#pragma unroll
  for (int b = -1; b <= 1; ++b)
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const double w = full_weight(b, fx) * (1.0 / fy);
      if (w != 0.0 && a < fy) s += w * By[df.at(clamp_index(fy * j + a, df.ny - 2), clamp_index(fx * i + b, df.nx - 1))];
    }
  return (double)(fx * fy) * s;
}
__device__ __forceinline__ void coarsen_point(const Dims& df, const Dims& dc, int fx, int fy, const double* Na,
                                              const double* Nb, const double* Bx, const double* By, double* cNa,
                                              double* cNb, double* cBx, double* cBy, int j, int i) {
  const long long q = dc.at(j, i);
  const bool jn = j < dc.ny - 1, in = i < dc.nx - 1;
  const double na = coarsen_Na(df, fx, fy, Na, j, i), nb = jn && in ? coarsen_Nb(df, fx, fy, Nb, j, i) : 0.0;
  const double bx = in ? coarsen_Bx(df, fx, fy, Bx, j, i) : 0.0, by = jn ? coarsen_By(df, fx, fy, By, j, i) : 0.0;
  cNa[q] = na;
  if (jn && in) cNb[q] = nb;
  if (in) cBx[q] = bx;
  if (jn) cBy[q] = by;
}

// the row types of the finest level from the SICO masks (assembly loop :1683-1727)
__global__ void k_row_types(Dims d, const int* combi, const int* inner, const int* outer, int8_t* rtu,
                            int8_t* rtv) {
  IDX2D
  if (j >= d.ny || i >= d.nx) return;
  const long long q = d.at(j, i);
  int8_t t = RT_FREE;
  if (u_int(d, j, i)) {
    const long long q1 = d.at(j, i + 1);
    if ((combi[q] == 3 && combi[q1] == 1) || (combi[q] == 1 && combi[q1] == 3)) {
      t = RT_IDENT;   // shelf next to land
    } else if ((inner[q] == 1 && outer[q1] == 1) || (outer[q] == 1 && inner[q1] == 1)) {
      const int i1 = inner[q] == 1 ? i : i + 1;
      if (outer[d.at(j, i1 - 1)] == 1 && outer[d.at(j, i1 + 1)] == 1) t = RT_IDENT;
      else t = i1 == i ? RT_MARGIN_LO : RT_MARGIN_HI;
    }
  }
  rtu[q] = t;
  t = RT_FREE;
  if (v_int(d, j, i)) {
    const long long q1 = d.at(j + 1, i);
    if ((combi[q] == 3 && combi[q1] == 1) || (combi[q] == 1 && combi[q1] == 3)) {
      t = RT_IDENT;
    } else if ((inner[q] == 1 && outer[q1] == 1) || (outer[q] == 1 && inner[q1] == 1)) {
      const int j1 = inner[q] == 1 ? j : j + 1;
      if (outer[d.at(j1 - 1, i)] == 1 && outer[d.at(j1 + 1, i)] == 1) t = RT_IDENT;
      else t = j1 == j ? RT_MARGIN_LO : RT_MARGIN_HI;
    }
  }
  rtv[q] = t;
}

// rhs of the free rows of the finest level (k_rhs), folded into the first set-up launch;
// with 'BC' margins, 0 for u = 0 rows and the front stress for front rows
struct RhsArgs {
  int on, crossterms;
  const double *tdx, *tdy, *Ncx, *Ncy;
  double *bu, *bv;
  const int8_t *rtu, *rtv;
  const double *Hi, *SL, *Hb;
};

// vertically integrated stress difference across a calving front at the ice cell q
// (0.5 rho_i g H^2 - 0.5 rho_sw g H_ocean^2, :2251-2262)
__device__ __forceinline__ double front_stress(const RhsArgs& r, long long q) {
  const double H = r.Hi[q];
  const double Ho = r.SL[q] > r.Hb[q] ? min_ref(kRhoI / kRhoSW * H, r.SL[q] - r.Hb[q]) : 0.0;
  return 0.5 * kRhoI * kGrav * H * H - 0.5 * kRhoSW * kGrav * Ho * Ho;
}

// Operator set-up of one level in one launch over its points: the inverse diagonals of
// level l, the rediscretised coefficients of level l+1 (coarse points are a subset of
// the fine index range) and, on the finest level, the right-hand side.
// float copies of the finest level's coefficients and inverse diagonals (DIVA_PREC_MIXED)
struct F32Out {
  float *Na, *Nb, *Bx, *By, *idu, *idv;
};

__global__ void k_level_setup(Op o, int coarsen, Dims dc, int fx, int fy, double* cNa, double* cNb, double* cBx,
                              double* cBy, double* idu, double* idv, RhsArgs rhs, F32Out f32) {
  IDX2D
  if (j >= o.d.ny || i >= o.d.nx) return;
  const long long q = o.d.at(j, i);
  // every load before the first store
  const bool ui = u_int(o.d, j, i), vi = v_int(o.d, j, i);
  const double iu = ui ? 1.0 / diag_u(o, j, i) : 0.0, iv = vi ? 1.0 / diag_v(o, j, i) : 0.0;
  double b0 = 0.0, b1 = 0.0;
  if (rhs.on) {
    const double dx2 = o.d.dx * o.d.dx;
    if (ui) b0 = rhs.crossterms ? -rhs.tdx[q] * dx2 : -rhs.tdx[q] * dx2 / rhs.Ncx[q];
    if (vi) b1 = rhs.crossterms ? -rhs.tdy[q] * dx2 : -rhs.tdy[q] * dx2 / rhs.Ncy[q];
    if (rhs.rtu) {
      const int tu = rhs.rtu[q], tv = rhs.rtv[q];
      if (tu == RT_IDENT) b0 = 0.0;
      else if (tu != RT_FREE) b0 = front_stress(rhs, o.d.at(j, tu == RT_MARGIN_LO ? i : i + 1));
      if (tv == RT_IDENT) b1 = 0.0;
      else if (tv != RT_FREE) b1 = front_stress(rhs, o.d.at(tv == RT_MARGIN_LO ? j : j + 1, i));
    }
  }
  const double na = f32.Na ? o.Na[q] : 0.0, nb = f32.Na ? o.Nb[q] : 0.0, bx = f32.Na ? o.Bx[q] : 0.0, by = f32.Na ? o.By[q] : 0.0;
  if (coarsen && j < dc.ny && i < dc.nx)   // (its loads, then its stores: other planes than those below)
    coarsen_point(o.d, dc, fx, fy, o.Na, o.Nb, o.Bx, o.By, cNa, cNb, cBx, cBy, j, i);
  idu[q] = iu;
  idv[q] = iv;
  if (f32.Na) {
    f32.Na[q] = (float)na;
    f32.Nb[q] = (float)nb;
    f32.Bx[q] = (float)bx;
    f32.By[q] = (float)by;
    f32.idu[q] = (float)iu;
    f32.idv[q] = (float)iv;
  }
  if (rhs.on) {
    rhs.bu[q] = b0;
    rhs.bv[q] = b1;
  }
}

// Operator set-up of the sub-cycle levels in one block: the first level's coefficients copied
// to shared memory, the coarser ones' formed there level by level (a thread per point and
// plane, one barrier per level), then every level's inverse diagonals at once, and the coarsest
// level's matrix and its inverse.  The same per-point operations as k_level_setup.  Bound by the
// latency of its phases: with each level's coefficients and diagonals read back from L2 level
// by level it took 41 us on 65 x 9 points and 52 us on 36 x 21, now 21 and 28 us.
struct SmallSetup {
  int first, last;           // the levels handled
  int direct;                // assemble and invert the coarsest level's matrix
  // when: 0 every launch; 1 in the viscosity iterations coarse_inverse_due() picks, read from
  // the device iteration counter (graph-launched loop); 2 not in this launch
  int inv_when;
  const double* sc;
  CoarseMap map;
  const uint16_t* tab;       // the coarsest level's row table
  double* Ainv;
  int* singular;
  Op o[kMaxLevels];
  double *idu[kMaxLevels], *idv[kMaxLevels];
  int fx[kMaxLevels], fy[kMaxLevels];
};

__global__ void __launch_bounds__(kInvThreads) k_small_setup(const __grid_constant__ SmallSetup a) {
  extern __shared__ double sm[];   // per level compact planes of N_a, N_b, B_x, B_y; two matrices of the inverse
  const int tid = threadIdx.x, lo = min(a.first, a.last);
  auto points = [&](int l) { return a.o[l].d.nx * a.o[l].d.ny; };
  auto compact = [&](int l, double* p) {   // level l's operator reading its planes at p
    Op o = a.o[l];
    o.d.ld = o.d.ny;
    const int n = points(l);
    o.Na = p; o.Nb = p + n; o.Bx = p + 2 * n; o.By = p + 3 * n;
    return o;
  };
  const int n0 = points(lo);
  for (int t = tid; t < n0; t += kInvThreads) {
    const Op& o = a.o[lo];
    const long long q = o.d.at(t % o.d.ny, t / o.d.ny);
    copy8(sm + t, o.Na + q);
    copy8(sm + n0 + t, o.Nb + q);
    copy8(sm + 2 * n0 + t, o.Bx + q);
    copy8(sm + 3 * n0 + t, o.By + q);
  }
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  double* p = sm;
  for (int l = lo; l < a.last; ++l) {   // a thread per coarse point and plane
    const Op f = compact(l, p);
    const int n = points(l), m = points(l + 1), ny = a.o[l + 1].d.ny, nx = a.o[l + 1].d.nx, fx = a.fx[l], fy = a.fy[l];
    double* k = p + 4 * n;
    for (int e = tid; e < 4 * m; e += kInvThreads) {
      const int plane = e / m, t = e - plane * m, j = t % ny, i = t / ny;
      const bool jn = j < ny - 1, in = i < nx - 1;
      double v = 0.0;
      if (plane == 0) v = coarsen_Na(f.d, fx, fy, f.Na, j, i);
      else if (plane == 1) { if (jn && in) v = coarsen_Nb(f.d, fx, fy, f.Nb, j, i); }
      else if (plane == 2) { if (in) v = coarsen_Bx(f.d, fx, fy, f.Bx, j, i); }
      else if (jn) v = coarsen_By(f.d, fx, fy, f.By, j, i);
      k[e] = v;
      if (plane == 0 || (plane == 1 ? jn && in : plane == 2 ? in : jn)) {
        const Op& o = a.o[l + 1];
        const_cast<double*>(plane == 0 ? o.Na : plane == 1 ? o.Nb : plane == 2 ? o.Bx : o.By)[o.d.at(j, i)] = v;
      }
    }
    __syncthreads();
    p = k;
  }
  // inverse diagonals of all levels
  int total = 0;
  for (int l = a.first; l <= a.last; ++l) total += 2 * points(l);
  for (int e = tid; e < total; e += kInvThreads) {
    int l = a.first, t = e;
    double* q = sm;
    while (t >= 2 * points(l)) { t -= 2 * points(l); q += 4 * points(l); ++l; }
    const Op o = compact(l, q);
    const int n = points(l);
    const bool u = t < n;
    if (!u) t -= n;
    const int j = t % o.d.ny, i = t / o.d.ny;
    const long long at = a.o[l].d.at(j, i);
    if (u) a.idu[l][at] = u_int(o.d, j, i) ? 1.0 / diag_u(o, j, i) : 0.0;
    else a.idv[l][at] = v_int(o.d, j, i) ? 1.0 / diag_v(o, j, i) : 0.0;
  }
  const bool inv = a.inv_when == 0 || (a.inv_when == 1 && coarse_inverse_due((int)a.sc[SC_PIC_IT]));
  if (a.direct && inv) coarse_setup_block(compact(a.last, p), a.map, a.tab, p + 4 * points(a.last), a.Ainv, a.singular);
}

// ---- Krylov kernels (fine level) --------------------------------------------------
// Every kernel with an inner product walks the points in 32 x 8 tiles with at most
// kRedBlocks blocks and finishes its reductions and the scalar step that follows itself
// (reduce_all): a reduction kernel and a one-thread control kernel of their own cost two
// launches of a few microseconds each, several times per Krylov half step (561 x 321: one
// viscosity iteration of 41 launches in 383 us).

constexpr int kPW = 3;   // inner products per kernel

// whether every value the u and v rows at (j,i) read is interior, so stored reads suffice
__device__ __forceinline__ bool rows_deep(const Dims& d, int j, int i) {
  return i >= 2 && i <= d.nx - 4 && j >= 2 && j <= d.ny - 4;
}
// (A x) of the interior u (v) row at (j,i): stored reads inside, the boundary mapping only
// next to it (the mapping's index selection for nine reads made the operator's kernels
// instruction-bound: k_matvec took 82 us on 1501 x 1501 for 22 us worth of bytes)
__device__ __forceinline__ double Au_any(const Op& o, const double* xu, const double* xv, int j, int i, bool deep) {
  return deep ? Au<true>(o, xu, xv, j, i) : Au(o, xu, xv, j, i);
}
__device__ __forceinline__ double Av_any(const Op& o, const double* xu, const double* xv, int j, int i, bool deep) {
  return deep ? Av<true>(o, xu, xv, j, i) : Av(o, xu, xv, j, i);
}

// out = A x ; dots [0] w.out, [1] out.out ; then the scalar step
enum { ST_NONE = 0, ST_ALPHA, ST_OMEGA };
// (Four blocks per SM: at the compiler's own choice of 98 registers two fit, too few loads in
// flight; with kRedBlocks 90 -> 55 us on 1501 x 1501, 14.5 -> 12.4 us on 321 x 561.)
__global__ void __launch_bounds__(256, 4) k_matvec(Op o, const double* xu, const double* xv, double* ou, double* ov,
                                                const double* wu, const double* wv, Reduction red, double* sc,
                                                int stage) {
  double acc[kPW] = {};
  FOR_TILES(o.d) {
    const long long q = o.d.at(j, i);
    const bool deep = rows_deep(o.d, j, i);
    double a = 0.0, b = 0.0;
    if (u_int(o.d, j, i)) {
      a = Au_any(o, xu, xv, j, i, deep);
      acc[0] += wu[q] * a;
      acc[1] += a * a;
    }
    if (v_int(o.d, j, i)) {
      b = Av_any(o, xu, xv, j, i, deep);
      acc[0] += wv[q] * b;
      acc[1] += b * b;
    }
    ou[q] = a;
    ov[q] = b;
  }
  if (!reduce_all(acc, red)) return;
  if (stage == ST_ALPHA) sc[SC_ALPHA] = acc[0] != 0.0 ? sc[SC_RHO] / acc[0] : 0.0;
  if (stage == ST_OMEGA) sc[SC_OMEGA] = acc[1] != 0.0 ? acc[0] / acc[1] : 0.0;
}

// The start of a viscosity iteration's linear solve: x <- (u, v), r = rhat = p = b - A x on
// the interior, and (raw) the nonlinear residual over all rows of the reference matrix, whose
// interior rows read stored values and whose boundary rows are u_src - u_b (or -u_b for zero).
// Dots: [0] raw r.r, [1] b.b, [2] r.r.
struct RelresTest {   // the stop test of a graph-launched iteration (h: IF(solve)), on = 0: none
  int on, stall_its;
  double tol;
  cudaGraphConditionalHandle h;
};
// (Every load of a point before its first store: the compiler moves none over a store.)
__global__ void __launch_bounds__(256, 4) k_init_residual(Op o, const double* u, const double* v, const double* bu,
                                                       const double* bv, double* xu, double* xv, double* ru,
                                                       double* rv, double* hu, double* hv, double* pu, double* pv,
                                                       int raw, Reduction red, double* sc, RelresTest test) {
  double acc[kPW] = {};
  FOR_TILES(o.d) {
    const long long q = o.d.at(j, i);
    const bool deep = rows_deep(o.d, j, i);
    const double u0 = u[q], v0 = v[q];
    double r0 = 0.0, w0 = 0.0, b0 = 0.0, r1 = 0.0, w1 = 0.0, b1 = 0.0;
    if (u_int(o.d, j, i)) {
      b0 = bu[q];
      r0 = b0 - Au_any(o, u, v, j, i, deep);
      w0 = (deep || !raw) ? r0 : b0 - Au<true>(o, u, v, j, i);
    } else if (raw && i < o.d.nx - 1) {
      w0 = LU(o, u, j, i) - u0;
    }
    if (v_int(o.d, j, i)) {
      b1 = bv[q];
      r1 = b1 - Av_any(o, u, v, j, i, deep);
      w1 = (deep || !raw) ? r1 : b1 - Av<true>(o, u, v, j, i);
    } else if (raw && j < o.d.ny - 1) {
      w1 = LV(o, v, j, i) - v0;
    }
    acc[0] += w0 * w0;
    acc[1] += b0 * b0;
    acc[2] += r0 * r0;
    acc[0] += w1 * w1;
    acc[1] += b1 * b1;
    acc[2] += r1 * r1;
    xu[q] = u0; ru[q] = r0; hu[q] = r0; pu[q] = r0;
    xv[q] = v0; rv[q] = r1; hv[q] = r1; pv[q] = r1;
  }
  if (!reduce_all(acc, red)) return;
  const double rr = acc[0], bb = acc[1];
  sc[SC_RR] = rr;
  sc[SC_BNORM2] = bb;
  sc[SC_RNORM2] = acc[2];
  sc[SC_RHO] = acc[2];
  if (!test.on) return;
  // nonlinear residual of the current iterate; skip the solve when it meets the tolerance
  const double relres = bb > 0.0 ? sqrt(rr / bb) : sqrt(rr);
  sc[SC_RELRES] = relres;
  sc[SC_ETA] = eta_after(sc[SC_ETA], relres, sc[SC_RELRES_PREV], test.tol);
  sc[SC_RELRES_PREV] = relres;
  bool stop = false;
  if (!isfinite(relres)) { sc[SC_NAN] = 1.0; stop = true; }
  else if (relres <= test.tol) { sc[SC_EXIT_RELRES] = 1.0; stop = true; }
  else if (stall_after(relres, sc + SC_STALL_BEST, sc + SC_STALL_SINCE, test.stall_its)) {
    sc[SC_EXIT_RELRES] = 1.0;   // ends like a converged one (basal stress at this state), flagged
    sc[SC_STALLED] = 1.0;
    stop = true;
  }
  cudaGraphSetConditional(test.h, stop ? 0u : 1u);
}

// Handles a kernel sets when it runs inside a graph-launched loop (on = 0: host-driven).
struct LoopHandles {
  int on;
  cudaGraphConditionalHandle a, b;
};

// s = r - alpha v ; dot [0] s.s ; then the half-step test: stop there if |s| meets the target
__global__ void __launch_bounds__(256) k_update_s(Dims d, double* sc, const double* ru, const double* rv,
                                                  const double* vu, const double* vv, double* su, double* sv,
                                                  Reduction red, LoopHandles h) {   // h.a: WHILE(krylov), h.b: IF(second)
  double acc[kPW] = {};
  const double alpha = sc[SC_ALPHA];
  FOR_TILES(d) {
    const long long q = d.at(j, i);
    const double a = ru[q] - alpha * vu[q], b = rv[q] - alpha * vv[q];
    su[q] = a;
    sv[q] = b;
    acc[0] += a * a;
    acc[0] += b * b;
  }
  if (!reduce_all(acc, red)) return;
  const double ss = acc[0];
  sc[SC_SNORM2] = ss;
  if (!h.on) return;
  sc[SC_LIN_IT] += 1.0;
  const bool fin = isfinite(ss), late = sc[SC_TIMEOUT] != 0.0, done = fin && !late && ss <= sc[SC_TARGET2];
  if (!fin) sc[SC_NAN] = 1.0;
  sc[SC_HALFDONE] = done ? 1.0 : 0.0;
  if (done) sc[SC_RNORM2] = ss;
  const bool go = fin && !late && !done;
  cudaGraphSetConditional(h.b, go ? 1u : 0u);
  if (!go) cudaGraphSetConditional(h.a, 0u);
}

// x += alpha phat + omega shat ; r = s - omega t ; dots [0] rhat.r, [1] r.r ; then rho, beta
// and the continue test
__global__ void __launch_bounds__(256) k_update_xr(Dims d, double* sc, double* xu, double* xv, const double* phu,
                                                   const double* phv, const double* shu, const double* shv,
                                                   const double* su, const double* sv, const double* tu,
                                                   const double* tv, double* ru, double* rv, const double* hu,
                                                   const double* hv, Reduction red, int maxit, LoopHandles h) {
  double acc[kPW] = {};
  const double alpha = sc[SC_ALPHA], omega = sc[SC_OMEGA];
  FOR_TILES(d) {
    const long long q = d.at(j, i);
    const bool ui = u_int(d, j, i), vi = v_int(d, j, i);
    double x0 = 0.0, r0 = 0.0, h0 = 0.0, x1 = 0.0, r1 = 0.0, h1 = 0.0;   // (loads before stores)
    if (ui) {
      x0 = xu[q] + (alpha * phu[q] + omega * shu[q]);
      r0 = su[q] - omega * tu[q];
      h0 = hu[q];
    }
    if (vi) {
      x1 = xv[q] + (alpha * phv[q] + omega * shv[q]);
      r1 = sv[q] - omega * tv[q];
      h1 = hv[q];
    }
    if (ui) {
      xu[q] = x0;
      ru[q] = r0;
      acc[0] += h0 * r0;
      acc[1] += r0 * r0;
    }
    if (vi) {
      xv[q] = x1;
      rv[q] = r1;
      acc[0] += h1 * r1;
      acc[1] += r1 * r1;
    }
  }
  if (!reduce_all(acc, red)) return;
  const double rho_new = acc[0], rr = acc[1], rho = sc[SC_RHO];
  sc[SC_BETA] = (rho != 0.0 && omega != 0.0) ? (rho_new / rho) * (alpha / omega) : 0.0;
  sc[SC_RHO] = rho_new;
  sc[SC_RNORM2] = rr;
  if (!h.on) return;
  sc[SC_LIN_FULL] += 1.0;
  const bool fin = isfinite(rr);
  if (!fin) sc[SC_NAN] = 1.0;
  const bool late = sc[SC_TIMEOUT] != 0.0;
  cudaGraphSetConditional(h.a, (fin && !late && rr > sc[SC_TARGET2] && sc[SC_LIN_IT] < (double)maxit) ? 1u : 0u);
}

// p = r + beta (p - omega v)
__global__ void k_update_p(Dims d, const double* sc, const double* ru, const double* rv, const double* vu,
                           const double* vv, double* pu, double* pv) {
  IDX2D
  if (j >= d.ny || i >= d.nx) return;
  const long long q = d.at(j, i);
  const double beta = sc[SC_BETA], omega = sc[SC_OMEGA];
  const double a = ru[q] + beta * (pu[q] - omega * vu[q]), b = rv[q] + beta * (pv[q] - omega * vv[q]);
  pu[q] = a;
  pv[q] = b;
}

// The solution of a linear solve: x, plus alpha phat when it ended at a half step (half 1; 0:
// not; -1: as the device scalar says), boundary unknowns from their sources.
__global__ void k_finish_x(Dims d, BCs bc, const double* sc, int half, const double* xu, const double* xv,
                           const double* phu, const double* phv, double* fu, double* fv) {
  IDX2D
  if (j >= d.ny || i >= d.nx) return;
  const bool add = half < 0 ? sc[SC_HALFDONE] != 0.0 : half != 0;
  const double alpha = sc[SC_ALPHA];
  const long long q = d.at(j, i);
  int js, is;
  double a = 0.0, b = 0.0;
  if (i < d.nx - 1 && u_src(d, bc, j, i, js, is)) {
    const long long p = d.at(js, is);
    a = xu[p];
    if (add) a += alpha * phu[p];
  }
  if (j < d.ny - 1 && v_src(d, bc, j, i, js, is)) {
    const long long p = d.at(js, is);
    b = xv[p];
    if (add) b += alpha * phv[p];
  }
  fu[q] = a;
  fv[q] = b;
}

// the target of this linear solve, and whether it needs any iteration
__global__ void k_ctl_lin_init(double* sc, cudaGraphConditionalHandle h_while, int adaptive, double lin_rtol,
                               int maxit) {
  const double rr = sc[SC_RNORM2], bb = sc[SC_BNORM2];
  double rtol = lin_rtol;
  if (adaptive) rtol = max_ref(lin_rtol, sc[SC_ETA] * min_ref(1.0, sc[SC_RELRES]));
  const double t = rtol * (bb > 0.0 ? sqrt(bb) : 1.0);
  sc[SC_TARGET2] = t * t;
  sc[SC_SOLVED] = 1.0;
  sc[SC_HALFDONE] = 0.0;
  if (!isfinite(rr)) sc[SC_NAN] = 1.0;
  cudaGraphSetConditional(h_while, (isfinite(rr) && rr > t * t && maxit > 0) ? 1u : 0u);
}

// ---- host side --------------------------------------------------------------------
Op op_of(const Ctx* c, int l) {
  Op o;
  o.d = c->lv[l].d;
  o.bc = c->bc;
  o.ax = c->lv[l].d.dx;   // placeholders, set below
  o.ay = 1.0;
  o.Na = c->lv[l].Na; o.Nb = c->lv[l].Nb; o.Bx = c->lv[l].Bx; o.By = c->lv[l].By;
  o.inv_dx = 1.0 / c->lv[l].d.dx;
  o.rtu = nullptr;
  o.rtv = nullptr;
  if (l == 0 && c->c.choice_ice_margin == DIVA_MARGIN_BC) {
    o.rtu = c->rtu;
    o.rtv = c->rtv;
  }
  return o;
}

}  // namespace

// per-level cell aspect ratio (hy/hx): kept in Level via d.dx (hx) and a side table
static double level_ax(const Ctx* c, int l) {
  double hx = c->d.dx, hy = c->d.dx;
  for (int q = 1; q <= l; ++q) {
    if (c->lv[q].d.nx != c->lv[q - 1].d.nx) hx *= 2.0;
    if (c->lv[q].d.ny != c->lv[q - 1].d.ny) hy *= 2.0;
  }
  return hy / hx;
}
static Op make_op(const Ctx* c, int l) {
  Op o = op_of(c, l);
  o.ax = level_ax(c, l);
  o.ay = 1.0 / o.ax;
  return o;
}
// The finest level of the mixed-precision preconditioner (DIVA_PREC_MIXED): its smoother runs
// in float on float copies of the coefficients and inverse diagonals (written by the
// finest level's set-up), with the pre-smoothed x and the residual stored as float in
// the level's tu/tv and ru/rv planes.  Everything else stays double.
static int sub_first_level(const Ctx* c);
static bool level_fp32(const Ctx* c, int l) {
  return c->c.precision == DIVA_PREC_MIXED && c->tiled && l < sub_first_level(c);
}
static OpT<float> make_op32(const Ctx* c, int l) {
  const Op o = make_op(c, l);
  OpT<float> f;
  f.d = o.d; f.bc = o.bc; f.ax = o.ax; f.ay = o.ay; f.inv_dx = o.inv_dx; f.rtu = o.rtu; f.rtv = o.rtv;
  f.Na = c->f32[l][F32_NA]; f.Nb = c->f32[l][F32_NB]; f.Bx = c->f32[l][F32_BX]; f.By = c->f32[l][F32_BY];
  return f;
}

static void factors(const Ctx* c, int l, int* fx, int* fy) {
  *fx = (c->lv[l + 1].d.nx != c->lv[l].d.nx) ? 2 : 1;
  *fy = (c->lv[l + 1].d.ny != c->lv[l].d.ny) ? 2 : 1;
}

#define GL(l) grid2d(c->lv[l].d.ny, c->lv[l].d.nx), block2d(), 0, c->stream

static CoarseMap coarse_map(const Ctx* c) {
  const Dims& d = c->lv[c->nlev - 1].d;
  CoarseMap m;
  m.ny = d.ny;
  m.nu = (d.nx > 3 && d.ny > 2) ? (d.nx - 3) * (d.ny - 2) : 0;
  m.nv = (d.nx > 2 && d.ny > 3) ? (d.nx - 2) * (d.ny - 3) : 0;
  return m;
}

static int coarse_direct_n(const Ctx* c) {
  const int n = coarse_map(c).n();
  return n > 0 && n <= kCoarseDirectMax ? n : 0;
}

static int sub_first_level(const Ctx* c);

int solver_setup(Ctx* c, int inv_when) {
  const diva_config_t& C = c->c;
  // the 'BC' front rows live on the finest level only; a grid too small to coarsen
  // would hand that level to the coarse direct solve, whose matrix has no front rows
  if (C.choice_ice_margin == DIVA_MARGIN_BC && c->nlev < 2)
    return set_error(c, DIVA_UNSUPPORTED, "choice_ice_margin 'BC' needs nx or ny of at least 9");
  if (C.precision == DIVA_PREC_MIXED && (c->nlev < 2 || !c->tiled))
    return set_error(c, DIVA_UNSUPPORTED,
                     "precision 'mixed' needs the tiled smoother (no periodic boundary, DIVA_NO_TILES unset) and nx or ny >= 9");
  // level l's diagonal and level l+1's coefficients in one launch; the finest level's
  // launch also forms the right-hand side, so it always runs on its own
  const int first_small = sub_first_level(c) > 1 ? sub_first_level(c) : 1;
  for (int l = 0; l < first_small && l < c->nlev; ++l) {
    const Level& F = c->lv[l];
    const bool coarsen = l + 1 < c->nlev;
    const Level& K = c->lv[coarsen ? l + 1 : l];
    int fx = 1, fy = 1;
    if (coarsen) factors(c, l, &fx, &fy);
    RhsArgs rhs{};
    if (l == 0) {
      rhs.on = 1;
      rhs.crossterms = C.include_SSADIVA_crossterms;
      rhs.tdx = c->D(DIVA_F_TAUDX_CX); rhs.tdy = c->D(DIVA_F_TAUDY_CY);
      rhs.Ncx = c->D(DIVA_F_N_CX); rhs.Ncy = c->D(DIVA_F_N_CY);
      rhs.bu = c->kv[KV_B][0]; rhs.bv = c->kv[KV_B][1];
      if (C.choice_ice_margin == DIVA_MARGIN_BC) {
        rhs.rtu = c->rtu; rhs.rtv = c->rtv;
        rhs.Hi = c->D(DIVA_F_HI_A); rhs.SL = c->D(DIVA_F_SL_A); rhs.Hb = c->D(DIVA_F_HB_A);
      }
    }
    F32Out f32{};
    if (level_fp32(c, l)) {
      float* const* f = c->f32[l];
      f32.Na = f[F32_NA]; f32.Nb = f[F32_NB]; f32.Bx = f[F32_BX]; f32.By = f[F32_BY];
      f32.idu = f[F32_IDU]; f32.idv = f[F32_IDV];
    }
    k_level_setup<<<GL(l)>>>(make_op(c, l), coarsen ? 1 : 0, K.d, fx, fy, K.Na, K.Nb, K.Bx, K.By, F.idu, F.idv,
                             rhs, f32); c->launches++;
    DIVA_LAUNCHED(c, "k_level_setup");
  }
  const CoarseMap m = coarse_map(c);
  c->coarse_n = m.nu + m.nv;
  c->coarse_direct = c->coarse_n > 0 && c->coarse_n <= kCoarseDirectMax;
  SmallSetup a{};
  a.first = first_small;
  a.last = c->nlev - 1;
  a.direct = c->coarse_direct ? 1 : 0;
  a.map = m;
  a.tab = c->sub_tab + c->sub_tab_off[c->nlev - 1];
  a.Ainv = c->coarse_inv;
  a.singular = c->coarse_singular;
  a.inv_when = inv_when;
  a.sc = c->scal;
  for (int l = a.first < a.last ? a.first : a.last; l <= a.last; ++l) {   // (first > last on a one-level grid)
    a.o[l] = make_op(c, l);
    a.idu[l] = c->lv[l].idu;
    a.idv[l] = c->lv[l].idv;
    a.fx[l] = a.fy[l] = 1;
    if (l < a.last) factors(c, l, &a.fx[l], &a.fy[l]);
  }
  size_t dbl = kInvDbl;
  for (int l = a.first < a.last ? a.first : a.last; l <= a.last; ++l) dbl += 4 * (size_t)c->lv[l].d.nx * c->lv[l].d.ny;
  k_small_setup<<<1, kInvThreads, dbl * sizeof(double), c->stream>>>(a); c->launches++;
  DIVA_LAUNCHED(c, "k_small_setup");
  return DIVA_OK;
}

static int gs_sweep(Ctx* c, int l, double* xu, double* xv, const double* bu, const double* bv, bool forward) {
  const Op o = make_op(c, l);
  const Level& L = c->lv[l];
  dim3 g = grid2d((L.d.ny + 1) / 2, L.d.nx);
  for (int p = 0; p < 4; ++p) {
    const int pp = forward ? p : 3 - p;
    k_gs<<<g, block2d(), 0, c->stream>>>(o, xu, xv, bu, bv, L.idu, L.idv, pp >> 1, pp & 1); c->launches++;
  }
  DIVA_LAUNCHED(c, "k_gs");
  c->fine_passes += (double)L.d.plane / (double)c->d.plane;
  return DIVA_OK;
}

// interior rows (u then v) of a level
static int level_rows(const Dims& d) {
  const int nu = (d.nx > 3 && d.ny > 2) ? (d.nx - 3) * (d.ny - 2) : 0;
  const int nv = (d.nx > 2 && d.ny > 3) ? (d.nx - 2) * (d.ny - 3) : 0;
  return nu + nv;
}

// Shared memory of the sub-cycle from level l down: the planes, the row tables, the inverse, the
// residual.  The level it starts from is the first whose planes, residual planes, reads and
// prolongation taps, and those of the levels below, fit in kSubSmemBudget (sub_bytes).
static size_t sub_points(const Ctx* c, int l) {
  size_t n = 0;
  for (int q = l; q < c->nlev; ++q) n += (size_t)c->lv[q].d.nx * c->lv[q].d.ny + 1;
  return n;
}
static size_t sub_rows(const Ctx* c, int l) {
  size_t n = 0;
  for (int q = l; q < c->nlev; ++q) n += ((size_t)(kTabReads + 1 + kTabProlong) * level_rows(c->lv[q].d) + 7) / 8 * 8;
  return n;
}
static int sub_first_fit(const Ctx* c);
// entries of a level's row table, padded to 8 (16 bytes) so that every level's table starts
// 16-byte aligned and the sub-cycle copies the tables as 16-byte vectors; the restriction
// taps only below the first level that may start the sub-cycle
static size_t level_tab_entries(const Ctx* c, int l) {
  const int R = level_rows(c->lv[l].d);
  return ((size_t)tab_restrict(R) + (l > sub_first_fit(c) ? kTabRestrict * R : 0) + 7) / 8 * 8;
}
static size_t sub_tab_entries(const Ctx* c, int l) {
  size_t n = 0;
  for (int q = l; q < c->nlev; ++q) n += level_tab_entries(c, q);
  return n;
}
// the coarsest level's unknowns when it is solved with its inverse, else 0
static int coarse_direct_n(const Ctx* c);
// doubles of the sub-cycle's table area (16-byte aligned), between the planes and the inverse
static size_t sub_tab_dbl(const Ctx* c, int l) { return ((sub_tab_entries(c, l) * sizeof(uint16_t) + 15) / 16) * 2; }
// doubles of the planes from level l down (an even number: the tables follow, 16-byte aligned)
static size_t sub_dbl(const Ctx* c, int l) { return (kSubArrays * sub_points(c, l) + 1) / 2 * 2; }
static size_t sub_bytes(const Ctx* c, int l) {
  const size_t n = (size_t)coarse_direct_n(c);
  return ((kSubArrays + 2) * sub_points(c, l) + (sub_rows(c, l) * sizeof(uint16_t) + 15) / 16 * 2 + n * n) * sizeof(double);
}
// what is allocated
static size_t sub_alloc(const Ctx* c, int l) {
  const size_t n = (size_t)coarse_direct_n(c);
  const Dims& d = c->lv[l].d;
  return (sub_dbl(c, l) + sub_tab_dbl(c, l) + n * n + 2 * ((size_t)d.nx * d.ny + 1)) * sizeof(double);
}

// the largest level whose levels all fit in the sub-cycle's shared memory (the row
// tables are built from there down, whatever the configuration)
static int sub_first_fit(const Ctx* c) {
  for (int l = 0; l < c->nlev; ++l)
    if (sub_bytes(c, l) <= kSubSmemBudget) return l;   // (then sub_alloc is at most kSubSmemMax)
  return c->nlev - 1;
}
// first level of the one-block sub-cycle
static int sub_first_level(const Ctx* c) {
  // the finest level's 'BC' front rows are not in the sub-cycle's row tables, and a
  // mixed-precision finest level is smoothed by the float tile kernels
  const bool own0 = c->c.choice_ice_margin == DIVA_MARGIN_BC || (c->c.precision == DIVA_PREC_MIXED && c->tiled);
  const int l0 = (own0 && c->nlev > 1) ? 1 : 0;
  const int f = sub_first_fit(c);
  return f > l0 ? f : l0;
}

static int vcycle(Ctx* c, int l, double* xu, double* xv, const double* bu, const double* bv,
                  const Restriction& rs);

// tile edge of level l's smoothing kernels, and whether they are 1.5x wider along i: by its size
// (tile_choice), unless the caller chose an edge (diva_set_tile_edges, e.g. from an autotuner)
static bool tile_chosen(const Ctx* c, int l) { return c->tile_override[l] == 16 || c->tile_override[l] == 32; }
static int tile_edge(const Ctx* c, int l) {
  return tile_chosen(c, l) ? c->tile_override[l] : tile_choice(c->lv[l].d.ny, c->lv[l].d.nx).edge;
}
static bool tile_wide(const Ctx* c, int l) {
  return !tile_chosen(c, l) && tile_choice(c->lv[l].d.ny, c->lv[l].d.nx).wide;
}

// Which tile kernels a level uses: the edge (tile_edge), and whether the region's
// coefficients are staged in shared memory (16 x 16 tiles: 92 KB, two blocks per SM;
// 32 x 32 tiles would need 200 KB, one block per SM, so they read the coefficients
// from L2 instead).
constexpr bool kStage16 = true, kStage32 = false;

// H: the tile's halo, 4 nu + 1 for nu sweeps per phase (halo_for); tiles of TJ rows (j)
// by TI columns (i)
template <int TJ, int TI, bool S, class R, int H>
static void tile_down_h(Ctx* c, int l, const OpT<R>& o, const R* idu, const R* idv, const Restriction& rs,
                        const double* bu, const double* bv, int nu) {
  const Level& L = c->lv[l];
  const dim3 grid((L.d.ny + TJ - 1) / TJ, (L.d.nx + TI - 1) / TI);
  // b is written only when it is restricted here (rs.on), which never happens on the finest level
  auto kern = o.rtu ? k_smooth_down<TJ, TI, S, true, R, H> : k_smooth_down<TJ, TI, S, false, R, H>;
  kern<<<grid, kTileThreads, TileGeom<TJ, TI, S, R, H>::smem, c->stream>>>(
      o, rs, const_cast<double*>(bu), const_cast<double*>(bv), reinterpret_cast<R*>(L.tu),
      reinterpret_cast<R*>(L.tv), reinterpret_cast<R*>(L.ru), reinterpret_cast<R*>(L.rv), idu, idv, nu);
  c->launches++;
}
template <int TJ, int TI, bool S, class R, int H>
static void tile_up_h(Ctx* c, int l, const OpT<R>& o, const R* idu, const R* idv, int fx, int fy, const double* bu,
                      const double* bv, double* xu, double* xv, int nu) {
  const Level& L = c->lv[l];
  const Level& K = c->lv[l + 1];
  const dim3 grid((L.d.ny + TJ - 1) / TJ, (L.d.nx + TI - 1) / TI);
  auto kern = o.rtu ? k_smooth_up<TJ, TI, S, true, R, H> : k_smooth_up<TJ, TI, S, false, R, H>;
  kern<<<grid, kTileThreads, TileGeom<TJ, TI, S, R, H>::smem_up, c->stream>>>(
      o, make_op(c, l + 1), fx, fy, K.xu, K.xv, bu, bv, reinterpret_cast<const R*>(L.tu),
      reinterpret_cast<const R*>(L.tv), xu, xv, idu, idv, nu);
  c->launches++;
}
template <int TJ, int TI, bool S, class R>
static void tile_down_r(Ctx* c, int l, const OpT<R>& o, const R* idu, const R* idv, const Restriction& rs,
                        const double* bu, const double* bv, int nu) {
  if (halo_for(nu) == kHaloOne) tile_down_h<TJ, TI, S, R, kHaloOne>(c, l, o, idu, idv, rs, bu, bv, nu);
  else tile_down_h<TJ, TI, S, R, kHalo>(c, l, o, idu, idv, rs, bu, bv, nu);
}
template <int TJ, int TI, bool S, class R>
static void tile_up_r(Ctx* c, int l, const OpT<R>& o, const R* idu, const R* idv, int fx, int fy, const double* bu,
                      const double* bv, double* xu, double* xv, int nu) {
  if (halo_for(nu) == kHaloOne) tile_up_h<TJ, TI, S, R, kHaloOne>(c, l, o, idu, idv, fx, fy, bu, bv, xu, xv, nu);
  else tile_up_h<TJ, TI, S, R, kHalo>(c, l, o, idu, idv, fx, fy, bu, bv, xu, xv, nu);
}
static int tile_down(Ctx* c, int l, const Restriction& rs, const double* bu, const double* bv, double* xu,
                     double* xv, int nu) {
  const Level& L = c->lv[l];
  const int T = tile_edge(c, l);
  const bool W = tile_wide(c, l);
  if (level_fp32(c, l)) {   // float tiles stage their coefficients at every shape (100 KB at 32 x 32)
    const OpT<float> o = make_op32(c, l);
    const float *iu = c->f32[l][F32_IDU], *iv = c->f32[l][F32_IDV];
    if (T == 32) W ? tile_down_r<32, 48, true>(c, l, o, iu, iv, rs, bu, bv, nu) : tile_down_r<32, 32, true>(c, l, o, iu, iv, rs, bu, bv, nu);
    else W ? tile_down_r<16, 24, true>(c, l, o, iu, iv, rs, bu, bv, nu) : tile_down_r<16, 16, true>(c, l, o, iu, iv, rs, bu, bv, nu);
  } else {
    const Op o = make_op(c, l);
    const double *iu = L.idu, *iv = L.idv;
    if (T == 32) W ? tile_down_r<32, 48, kStage32>(c, l, o, iu, iv, rs, bu, bv, nu) : tile_down_r<32, 32, kStage32>(c, l, o, iu, iv, rs, bu, bv, nu);
    else W ? tile_down_r<16, 24, kStage16>(c, l, o, iu, iv, rs, bu, bv, nu) : tile_down_r<16, 16, kStage16>(c, l, o, iu, iv, rs, bu, bv, nu);
  }
  DIVA_LAUNCHED(c, "k_smooth_down");
  return DIVA_OK;
}
static int tile_up(Ctx* c, int l, int fx, int fy, const double* bu, const double* bv, double* xu, double* xv,
                   int nu) {
  const Level& L = c->lv[l];
  const int T = tile_edge(c, l);
  const bool W = tile_wide(c, l);
  if (level_fp32(c, l)) {
    const OpT<float> o = make_op32(c, l);
    const float *iu = c->f32[l][F32_IDU], *iv = c->f32[l][F32_IDV];
    if (T == 32) W ? tile_up_r<32, 48, true>(c, l, o, iu, iv, fx, fy, bu, bv, xu, xv, nu) : tile_up_r<32, 32, true>(c, l, o, iu, iv, fx, fy, bu, bv, xu, xv, nu);
    else W ? tile_up_r<16, 24, true>(c, l, o, iu, iv, fx, fy, bu, bv, xu, xv, nu) : tile_up_r<16, 16, true>(c, l, o, iu, iv, fx, fy, bu, bv, xu, xv, nu);
  } else {
    const Op o = make_op(c, l);
    const double *iu = L.idu, *iv = L.idv;
    if (T == 32) W ? tile_up_r<32, 48, kStage32>(c, l, o, iu, iv, fx, fy, bu, bv, xu, xv, nu) : tile_up_r<32, 32, kStage32>(c, l, o, iu, iv, fx, fy, bu, bv, xu, xv, nu);
    else W ? tile_up_r<16, 24, kStage16>(c, l, o, iu, iv, fx, fy, bu, bv, xu, xv, nu) : tile_up_r<16, 16, kStage16>(c, l, o, iu, iv, fx, fy, bu, bv, xu, xv, nu);
  }
  DIVA_LAUNCHED(c, "k_smooth_up");
  return DIVA_OK;
}

// Whether level l is smoothed by the streamed kernel: double, two sweeps per phase, a size at which
// that pays, and no edge chosen by the caller.  Float levels keep the tiles, which hold the
// coefficients of a 32 x 32 tile in shared memory: 41 / 46 us at 321 x 561.
static int level_nu(const Ctx* c, int l);
static bool level_streamed(const Ctx* c, int l) {
  const Dims& d = c->lv[l].d;
  return !tile_chosen(c, l) && !level_fp32(c, l) && level_nu(c, l) == WaveGeom::NU && strips_pay(d.ny, d.nx);
}
template <bool UP>
static void launch_wave(Ctx* c, int l, const double* bu, const double* bv, double* ou, double* ov) {
  using G = WaveGeom;
  const Level& L = c->lv[l];
  WaveArgs a{};
  a.o = make_op(c, l);
  a.idu = L.idu; a.idv = L.idv; a.bu = bu; a.bv = bv;
  a.xu = L.tu; a.xv = L.tv; a.ru = L.ru; a.rv = L.rv;
  a.fail = c->scal + SC_TIMEOUT;
  a.drop = c->wave_drop;
  if (UP) {
    a.ou = ou; a.ov = ov;
    a.oc = make_op(c, l + 1);
    a.xcu = c->lv[l + 1].xu; a.xcv = c->lv[l + 1].xv;
    factors(c, l, &a.fx, &a.fy);
  }
  const WaveShape shape = wave_shape(L.d.ny, L.d.nx);
  a.rows = shape.rows;
  a.chunk = shape.chunk;
  const dim3 grid(shape.nstrip, shape.nchunk);
  const auto kern = a.o.rtu ? k_wave<true, UP> : k_wave<false, UP>;   // 'BC' rows: the finest level
  kern<<<grid, 32 * (UP ? G::warps_up : G::warps_down), UP ? G::smem_up : G::smem_down, c->stream>>>(a);
  c->launches++;
}
// pre-smoothing from x = 0 (the descent of a V-cycle enters every level with x = 0): two forward
// sweeps (u0 u1 v0 v1), x and r = b - A x written; b first, where it is the finer level's residual
static int wave_down(Ctx* c, int l, const Restriction& rs, const double* bu, const double* bv) {
  if (rs.on) {
    k_restrict_b<<<GL(l)>>>(rs.df, c->lv[l].d, rs.fx, rs.fy, static_cast<const double*>(rs.ru),
                            static_cast<const double*>(rs.rv), const_cast<double*>(bu), const_cast<double*>(bv));
    c->launches++;
    DIVA_LAUNCHED(c, "k_restrict_b");
  }
  launch_wave<false>(c, l, bu, bv, nullptr, nullptr);
  DIVA_LAUNCHED(c, "k_wave (descent)");
  return DIVA_OK;
}
// post-smoothing: x += P x_c, then two backward sweeps (v1 v0 u1 u0)
static int wave_up(Ctx* c, int l, const double* bu, const double* bv, double* xu, double* xv) {
  launch_wave<true>(c, l, bu, bv, xu, xv);
  DIVA_LAUNCHED(c, "k_wave (ascent)");
  return DIVA_OK;
}

// V-cycle step of a tiled level: 2 launches for the smoothing, the residual and the
// restriction instead of 4 per sweep and 2 more
static int vcycle_tiled(Ctx* c, int l, double* xu, double* xv, const double* bu, const double* bv,
                        const Restriction& rs, int nu1, int nu2) {
  if (4 * nu1 > halo_for(nu1) - 1 || 4 * nu2 > halo_for(nu2) - 1)
    return set_error(c, DIVA_UNSUPPORTED, "tiled smoothing depth");
  const Level& L = c->lv[l];
  const Level& K = c->lv[l + 1];
  const bool wave = level_streamed(c, l);
  int st = wave ? wave_down(c, l, rs, bu, bv) : tile_down(c, l, rs, bu, bv, xu, xv, nu1);
  if (st) return st;
  Restriction next{};
  next.on = 1;
  next.df = L.d;
  factors(c, l, &next.fx, &next.fy);
  next.ru = L.ru;
  next.rv = L.rv;
  next.rfloat = level_fp32(c, l) ? 1 : 0;   // the float residual of a mixed-precision level
  if ((st = vcycle(c, l + 1, K.xu, K.xv, K.bu, K.bv, next))) return st;
  if ((st = wave ? wave_up(c, l, bu, bv, xu, xv) : tile_up(c, l, next.fx, next.fy, bu, bv, xu, xv, nu2))) return st;
  c->fine_passes += (nu1 + nu2 + 1) * (double)L.d.plane / (double)c->d.plane;
  return DIVA_OK;
}

// Shared-memory limits of the tiled kernels (the 32 x 32 tiles need 80 KB) and of
// the sub-cycle, and whether the grid's boundary conditions allow tiles at all.
// Row tables of the sub-cycle levels (see k_subcycle), built on the host from the
// level sizes and the boundary conditions and copied to the context's table area.
static int build_sub_tables(Ctx* c) {
  const int first = sub_first_fit(c);
  std::vector<uint16_t> tab(sub_tab_entries(c, first));
  size_t off = 0;
  for (int l = first; l < c->nlev; ++l) {
    Dims d = c->lv[l].d;
    d.ld = d.ny;   // compact planes in shared memory
    const int P = d.nx * d.ny, R = level_rows(d);
    if (P + 1 >= 1 << kTapBits) return set_error(c, DIVA_UNSUPPORTED, "sub-cycle level too large for its row tables");
    c->sub_tab_off[l] = off;
    uint16_t *reads = tab.data() + off, *pos = reads + tab_pos(R), *prolong = reads + tab_prolong(R),
             *restricted = reads + tab_restrict(R);
    auto tap = [](size_t at, double w) { return (uint16_t)(at | (size_t)(16.0 * w - 1.0) << kTapBits); };
    int r = 0;
    auto put = [&](int j, int i, bool urow) {
      const int js_[4] = {urow ? j : j + 1, urow ? j : j - 1, urow ? j + 1 : j, urow ? j - 1 : j};
      const int is_[4] = {urow ? i + 1 : i, urow ? i - 1 : i, urow ? i : i + 1, urow ? i : i - 1};
      const int jc_[4] = {urow ? j : j + 1, urow ? j : j + 1, urow ? j - 1 : j, urow ? j - 1 : j};
      const int ic_[4] = {urow ? i : i - 1, urow ? i + 1 : i, urow ? i : i - 1, urow ? i + 1 : i};
      pos[r] = (uint16_t)d.at(j, i);
      for (int k = 0; k < 4; ++k) {   // same-component neighbours, then the cross-coupled reads
        int js, is;
        const bool on = urow ? u_src(d, c->bc, js_[k], is_[k], js, is) : v_src(d, c->bc, js_[k], is_[k], js, is);
        reads[8 * r + k] = on ? (uint16_t)d.at(js, is) : (uint16_t)P;
        const bool on2 = urow ? v_src(d, c->bc, jc_[k], ic_[k], js, is) : u_src(d, c->bc, jc_[k], ic_[k], js, is);
        reads[8 * r + 4 + k] = on2 ? (uint16_t)d.at(js, is) : (uint16_t)P;
      }
      // the prolongation taps of the row from the next level (prolong_delta's taps in its
      // order, each clamped and read through the coarse level's boundary mapping; the
      // coarse plane's zero element for a 'zero' side or a tap the row does not have)
      if (l + 1 < c->nlev) {
        Dims dc = c->lv[l + 1].d;
        dc.ld = dc.ny;
        const int Pc = dc.nx * dc.ny;
        int fx, fy;
        factors(c, l, &fx, &fy);
        int k = 0, js, is, Cj, Ci;
        double wj, wi;
        auto clampi = [](int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); };
        if (urow) {
          for (int a = 0; a < scatter_node_n(j, fy); ++a)
            for (int b = 0; b < scatter_cell_n(i, fx); ++b, ++k) {
              scatter_node(j, fy, a, Cj, wj);
              scatter_cell(i, fx, b, Ci, wi);
              const bool on = u_src(dc, c->bc, clampi(Cj, 0, dc.ny - 1), clampi(Ci, 0, dc.nx - 2), js, is);
              prolong[kTabProlong * r + k] = tap(on ? dc.at(js, is) : Pc, wj * wi);
            }
        } else {
          for (int a = 0; a < scatter_cell_n(j, fy); ++a)
            for (int b = 0; b < scatter_node_n(i, fx); ++b, ++k) {
              scatter_cell(j, fy, a, Cj, wj);
              scatter_node(i, fx, b, Ci, wi);
              const bool on = v_src(dc, c->bc, clampi(Cj, 0, dc.ny - 2), clampi(Ci, 0, dc.nx - 1), js, is);
              prolong[kTabProlong * r + k] = tap(on ? dc.at(js, is) : Pc, wj * wi);
            }
        }
        for (; k < kTabProlong; ++k) prolong[kTabProlong * r + k] = tap(Pc, 1.0);
      }
      // the restriction taps of the row from the level above (restrict_values' taps in its order),
      // one beyond the position; 0 for none
      if (l > first) {
        Dims df = c->lv[l - 1].d;
        df.ld = df.ny;
        int fx, fy, fj, fi, k = 0;
        double wj, wi;
        factors(c, l - 1, &fx, &fy);
        const int nj = urow ? gather_node_n(fy) : gather_cell_n(fy), ni = urow ? gather_cell_n(fx) : gather_node_n(fx);
        for (int a = 0; a < nj; ++a)
          for (int b = 0; b < ni; ++b) {
            if (urow) { gather_node(j, fy, a, fj, wj); gather_cell(i, fx, b, fi, wi); }
            else { gather_cell(j, fy, a, fj, wj); gather_node(i, fx, b, fi, wi); }
            if (urow ? u_int(df, fj, fi) : v_int(df, fj, fi))
              restricted[kTabRestrict * r + k++] = tap(df.at(fj, fi) + 1, wj * wi);
          }
      }
      ++r;
    };
    for (int p = 0; p < 4; ++p) {
      c->sub_cls[l][p] = r;
      const bool urow = p < 2;
      for (int i = 0; i < d.nx; ++i)
        for (int j = 0; j < d.ny; ++j)
          if (((i + j) & 1) == (p & 1) && (urow ? u_int(d, j, i) : v_int(d, j, i))) put(j, i, urow);
    }
    c->sub_cls[l][4] = r;
    if (r != R) return set_error(c, DIVA_CUDA_ERROR, "sub-cycle row table size");
    off += level_tab_entries(c, l);
  }
  if (!tab.empty())
    DIVA_CUDA(c, cudaMemcpy(c->sub_tab, tab.data(), tab.size() * sizeof(uint16_t), cudaMemcpyHostToDevice));
  return DIVA_OK;
}

size_t solver_table_entries(const Ctx* c) { return sub_tab_entries(c, sub_first_fit(c)); }

// dynamic shared memory of the four tile kernels (down/up, with/without front rows) of one shape
template <int TJ, int TI, bool S, class R, int H>
static int tile_attrs(Ctx* c) {
  using G = TileGeom<TJ, TI, S, R, H>;
  const void* k[4] = {(const void*)k_smooth_down<TJ, TI, S, false, R, H>, (const void*)k_smooth_down<TJ, TI, S, true, R, H>,
                      (const void*)k_smooth_up<TJ, TI, S, false, R, H>, (const void*)k_smooth_up<TJ, TI, S, true, R, H>};
  for (int q = 0; q < 4; ++q)   // the up kernels (2, 3) also stage the coarse correction
    DIVA_CUDA(c, cudaFuncSetAttribute(k[q], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(q < 2 ? G::smem : G::smem_up)));
  return DIVA_OK;
}
// every tile shape (square, and 1.5x wider along i) of both edges, both types, both halos
template <int TJ, int TI>
static int tile_attrs_shape(Ctx* c) {
  constexpr bool S = TJ == 16 ? kStage16 : kStage32;
  if (int st = tile_attrs<TJ, TI, S, double, kHalo>(c)) return st;
  if (int st = tile_attrs<TJ, TI, true, float, kHalo>(c)) return st;
  if (int st = tile_attrs<TJ, TI, S, double, kHaloOne>(c)) return st;
  if (int st = tile_attrs<TJ, TI, true, float, kHaloOne>(c)) return st;
  return DIVA_OK;
}

int solver_init(Ctx* c) {
  if (sub_bytes(c, c->nlev - 1) > kSubSmemBudget)
    return set_error(c, DIVA_UNSUPPORTED, "coarsest multigrid level too large for the one-block sub-cycle");
  if (int st = build_sub_tables(c)) return st;
  DIVA_CUDA(c, cudaFuncSetAttribute(k_small_setup, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSubSmemBudget));
  DIVA_CUDA(c, cudaFuncSetAttribute(k_subcycle, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSubSmemMax));
  if (int st = tile_attrs_shape<32, 32>(c)) return st;
  if (int st = tile_attrs_shape<16, 16>(c)) return st;
  if (int st = tile_attrs_shape<32, 48>(c)) return st;
  if (int st = tile_attrs_shape<16, 24>(c)) return st;
  const void* wave[4] = {(const void*)k_wave<false, false>, (const void*)k_wave<true, false>,
                         (const void*)k_wave<false, true>, (const void*)k_wave<true, true>};
  for (int q = 0; q < 4; ++q)
    DIVA_CUDA(c, cudaFuncSetAttribute(wave[q], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(q < 2 ? WaveGeom::smem_down : WaveGeom::smem_up)));
  const BCs& b = c->bc;
  const int all[8] = {b.uW, b.uE, b.uS, b.uN, b.vW, b.vE, b.vS, b.vN};
  bool periodic = false;
  for (int q = 0; q < 8; ++q) periodic = periodic || all[q] == DIVA_BC_PERIODIC;
  c->tiled = !periodic && !c->tiles_disabled;
  return DIVA_OK;
}

// One V-cycle from level l down, entered with x = 0.  b is given in bu/bv, or (rs.on)
// restricted from the finer level's residual by the level's first kernel.
// Gauss-Seidel sweeps before and after the coarse correction.  The finest level and every
// coarser level of at least DIVA_MG_NU2_POINTS points take two (V(2,2)); smaller levels,
// whose kernels are bound by the latency of their barrier-separated colour passes rather
// than by their points, take one (V(1,1)), and so does the one-block sub-cycle.  Measured
// on one B200, solves to rel-res 1e-6: on the 321 x 561 ice cap one sweep below the finest
// level keeps the V-cycle count of V(2,2) everywhere (79 relaxed, 43 with Anderson mixing)
// at 8-13 % less time per solve; on the 1501 x 1501 sheet one sweep on its large coarse
// levels (751 x 751, 376 x 376) doubled the V-cycles per viscosity iteration.
#ifndef DIVA_MG_NU2_POINTS
#define DIVA_MG_NU2_POINTS 100000
#endif
static int level_nu(const Ctx* c, int l) {
  return (l == 0 || (long long)c->lv[l].d.nx * c->lv[l].d.ny >= DIVA_MG_NU2_POINTS) ? 2 : 1;
}
static int vcycle(Ctx* c, int l, double* xu, double* xv, const double* bu, const double* bv,
                  const Restriction& rs) {
  const int nu1 = level_nu(c, l), nu2 = nu1, coarse_sweeps = 64;
  if (l == sub_first_level(c)) {
    SubCycle sc{};
    sc.first = l;
    sc.last = c->nlev - 1;
    sc.nu1 = nu1;
    sc.nu2 = nu2;
    sc.coarse_sweeps = coarse_sweeps;
    sc.direct = c->coarse_direct ? 1 : 0;
    sc.map = coarse_map(c);
    sc.Ainv = c->coarse_inv;
    sc.singular = c->coarse_singular;
    int soff = 0, toff = 0;
    for (int q = l; q < c->nlev; ++q) {
      const Level& L = c->lv[q];
      SubLevel& S = sc.L[q];
      S.o = make_op(c, q);
      S.idu = L.idu; S.idv = L.idv;
      S.soff = soff;
      soff += kSubArrays * (L.d.nx * L.d.ny + 1);
      S.rows = level_rows(L.d);
      for (int k = 0; k < 5; ++k) S.cls[k] = c->sub_cls[q][k];
      for (int k = 0; k < 4; ++k) S.most = std::max(S.most, S.cls[k + 1] - S.cls[k]);
      S.toff = toff;
      S.gtab = c->sub_tab + c->sub_tab_off[q];
      toff += (int)level_tab_entries(c, q);
    }
    sc.dbl = (int)sub_dbl(c, l);
    sc.ainv_off = sc.dbl + (int)sub_tab_dbl(c, l);
    sc.res_off = sc.ainv_off + coarse_direct_n(c) * coarse_direct_n(c);
    sc.tab16 = toff / 8;
    sc.rs = rs;
    k_subcycle<<<1, kSubThreads, sub_alloc(c, l), c->stream>>>(sc, xu, xv, bu, bv); c->launches++;
    DIVA_LAUNCHED(c, "k_subcycle");
    for (int q = l; q < c->nlev; ++q) c->fine_passes += 8.0 * (double)c->lv[q].d.plane / (double)c->d.plane;
    return DIVA_OK;
  }
  const Level& L = c->lv[l];
  const Level& K = c->lv[l + 1];
  int st;
  if (c->tiled) return vcycle_tiled(c, l, xu, xv, bu, bv, rs, nu1, nu2);
  for (int s = 0; s < nu1; ++s)
    if ((st = gs_sweep(c, l, xu, xv, bu, bv, true))) return st;
  k_residual<<<GL(l)>>>(make_op(c, l), xu, xv, bu, bv, L.ru, L.rv); c->launches++;
  DIVA_LAUNCHED(c, "k_residual");
  int fx, fy;
  factors(c, l, &fx, &fy);
  k_restrict<<<GL(l + 1)>>>(L.d, K.d, fx, fy, L.ru, L.rv, K.bu, K.bv, K.xu, K.xv); c->launches++;
  DIVA_LAUNCHED(c, "k_restrict");
  if ((st = vcycle(c, l + 1, K.xu, K.xv, K.bu, K.bv, Restriction{}))) return st;
  k_prolong<<<GL(l)>>>(make_op(c, l + 1), L.d, fx, fy, K.xu, K.xv, xu, xv); c->launches++;
  DIVA_LAUNCHED(c, "k_prolong");
  for (int s = 0; s < nu2; ++s)
    if ((st = gs_sweep(c, l, xu, xv, bu, bv, false))) return st;
  return DIVA_OK;
}

// z = M^{-1} r: one V-cycle from zero
static int precond(Ctx* c, const double* ru, const double* rv, double* zu, double* zv) {
  // the tiled kernels and the sub-cycle start from x = 0 themselves and write every
  // point of z; the per-colour sweeps read x
  if (!c->tiled && sub_first_level(c) > 0) {
    DIVA_CUDA(c, cudaMemsetAsync(zu, 0, sizeof(double) * c->d.plane, c->stream));
    DIVA_CUDA(c, cudaMemsetAsync(zv, 0, sizeof(double) * c->d.plane, c->stream));
  }
  c->mg_cycles++;
  return vcycle(c, 0, zu, zv, ru, rv, Restriction{});
}

static int read_scalars(Ctx* c) {
  DIVA_CUDA(c, cudaMemcpyAsync(c->h_scal, c->scal, sizeof(double) * SC_COUNT, cudaMemcpyDeviceToHost, c->stream));
  DIVA_CUDA(c, cudaStreamSynchronize(c->stream));
  return DIVA_OK;
}

static Reduction reduction(Ctx* c) { return Reduction{c->partials, c->red_count}; }

// x <- (u, v), the initial residual, its norms and (raw) the nonlinear residual's
static void launch_init_residual(Ctx* c, const double* u, const double* v, int raw, const RelresTest& test) {
  auto K = c->kv;
  k_init_residual<<<red_blocks(c->d), block2d(), 0, c->stream>>>(
      make_op(c, 0), u, v, K[KV_B][0], K[KV_B][1], K[KV_X][0], K[KV_X][1], K[KV_R][0], K[KV_R][1], K[KV_RHAT][0],
      K[KV_RHAT][1], K[KV_P][0], K[KV_P][1], raw, reduction(c), c->scal, test); c->launches++;
  c->fine_passes += 1.0;
}
// v = A phat and alpha, then s = r - alpha v and the half-step test (after the V-cycle p -> phat)
static void launch_first_half(Ctx* c, const LoopHandles& h) {
  auto K = c->kv;
  const int nb = red_blocks(c->d);
  k_matvec<<<nb, block2d(), 0, c->stream>>>(make_op(c, 0), K[KV_PHAT][0], K[KV_PHAT][1], K[KV_V][0], K[KV_V][1],
                                            K[KV_RHAT][0], K[KV_RHAT][1], reduction(c), c->scal, ST_ALPHA); c->launches++;
  k_update_s<<<nb, block2d(), 0, c->stream>>>(c->d, c->scal, K[KV_R][0], K[KV_R][1], K[KV_V][0], K[KV_V][1],
                                              K[KV_S][0], K[KV_S][1], reduction(c), h); c->launches++;
  c->fine_passes += 3.0;
}
// t = A shat and omega, x and r, rho and beta, p (after the V-cycle s -> shat)
static void launch_second_half(Ctx* c, const LoopHandles& h) {
  auto K = c->kv;
  const int nb = red_blocks(c->d);
  k_matvec<<<nb, block2d(), 0, c->stream>>>(make_op(c, 0), K[KV_SHAT][0], K[KV_SHAT][1], K[KV_T][0], K[KV_T][1],
                                            K[KV_S][0], K[KV_S][1], reduction(c), c->scal, ST_OMEGA); c->launches++;
  k_update_xr<<<nb, block2d(), 0, c->stream>>>(c->d, c->scal, K[KV_X][0], K[KV_X][1], K[KV_PHAT][0], K[KV_PHAT][1],
                                               K[KV_SHAT][0], K[KV_SHAT][1], K[KV_S][0], K[KV_S][1], K[KV_T][0],
                                               K[KV_T][1], K[KV_R][0], K[KV_R][1], K[KV_RHAT][0], K[KV_RHAT][1],
                                               reduction(c), c->c.lin_maxit, h); c->launches++;
  k_update_p<<<grid2d(c->d.ny, c->d.nx), block2d(), 0, c->stream>>>(c->d, c->scal, K[KV_R][0], K[KV_R][1], K[KV_V][0],
                                                                    K[KV_V][1], K[KV_P][0], K[KV_P][1]); c->launches++;
  c->fine_passes += 3.0;
}
// the solution (KV_XF)
static void launch_finish_x(Ctx* c, int half) {
  auto K = c->kv;
  k_finish_x<<<grid2d(c->d.ny, c->d.nx), block2d(), 0, c->stream>>>(c->d, c->bc, c->scal, half, K[KV_X][0], K[KV_X][1],
                                                                    K[KV_PHAT][0], K[KV_PHAT][1], K[KV_XF][0],
                                                                    K[KV_XF][1]); c->launches++;
}

int solver_solve(Ctx* c, const double* u0, const double* v0, double rtol, int maxit, int* iters, double* relres0) {
  auto U_ = [&](int k) { return c->kv[k][0]; };
  auto V_ = [&](int k) { return c->kv[k][1]; };
  launch_init_residual(c, u0, v0, 0, RelresTest{});
  DIVA_LAUNCHED(c, "k_init_residual");
  int st = read_scalars(c);
  if (st) return st;
  const double bnorm = sqrt(c->h_scal[SC_BNORM2]);
  double rnorm = sqrt(c->h_scal[SC_RNORM2]);
  if (relres0) *relres0 = bnorm > 0.0 ? rnorm / bnorm : rnorm;
  const double target = rtol * (bnorm > 0.0 ? bnorm : 1.0);
  int it = 0, half = 0;
  bool done = rnorm <= target;
  while (!done && it < maxit) {
    ++it;
    if ((st = precond(c, U_(KV_P), V_(KV_P), U_(KV_PHAT), V_(KV_PHAT)))) return st;
    launch_first_half(c, LoopHandles{});
    DIVA_LAUNCHED(c, "bicgstab half step");
    if ((st = read_scalars(c))) return st;
    if (c->h_scal[SC_TIMEOUT] != 0.0) return set_error(c, DIVA_TIMEOUT, kTimeoutMessage);
    if (sqrt(c->h_scal[SC_SNORM2]) <= target) {
      half = 1;
      rnorm = sqrt(c->h_scal[SC_SNORM2]);
      done = true;
      break;
    }
    if ((st = precond(c, U_(KV_S), V_(KV_S), U_(KV_SHAT), V_(KV_SHAT)))) return st;
    launch_second_half(c, LoopHandles{});
    DIVA_LAUNCHED(c, "bicgstab full step");
    if ((st = read_scalars(c))) return st;
    if (c->h_scal[SC_TIMEOUT] != 0.0) return set_error(c, DIVA_TIMEOUT, kTimeoutMessage);
    rnorm = sqrt(c->h_scal[SC_RNORM2]);
    if (!std::isfinite(rnorm)) return set_error(c, DIVA_NAN_DETECTED, "NaN in the linear solve");
    done = rnorm <= target;
  }
  launch_finish_x(c, half);
  DIVA_LAUNCHED(c, "k_finish_x");
  *iters = it;
  c->lin_iters += it;
  if (!done) {
    char buf[160];
    snprintf(buf, sizeof(buf), "linear solve reached %d iterations at relative residual %.3e (target %.1e)", it,
             bnorm > 0 ? rnorm / bnorm : rnorm, rtol);
    c->err = buf;
    return DIVA_LINEAR_NOT_CONVERGED;
  }
  return DIVA_OK;
}

int solver_relres(Ctx* c, const double* u, const double* v, double* relres) {
  launch_init_residual(c, u, v, 1, RelresTest{});
  DIVA_LAUNCHED(c, "k_init_residual");
  int st = read_scalars(c);
  if (st) return st;
  const double bb = c->h_scal[SC_BNORM2], rr = c->h_scal[SC_RR];
  *relres = bb > 0.0 ? sqrt(rr / bb) : sqrt(rr);
  return DIVA_OK;
}

// Fine-level smoothing as the V-cycle runs it (used to time the smoother): the tiled
// pre- and post-smoothing kernels (V(2,2), residual included) when the grid is tiled,
// else `sweeps` per-colour sweeps.  x, b and the coarse correction are the solver's
// scratch vectors.
int solver_smooth_fine(Ctx* c, int sweeps) {
  if (c->tiled && c->nlev > 1 && sub_first_level(c) > 0) {
    const int nu = 2;
    int fx, fy;
    factors(c, 0, &fx, &fy);
    double *xu = c->kv[KV_X][0], *xv = c->kv[KV_X][1];
    double *bu = c->kv[KV_B][0], *bv = c->kv[KV_B][1];   // not written: the restriction is off
    const bool wave = level_streamed(c, 0);
    int st = wave ? wave_down(c, 0, Restriction{}, bu, bv) : tile_down(c, 0, Restriction{}, bu, bv, xu, xv, nu);
    if (!st) st = wave ? wave_up(c, 0, bu, bv, xu, xv) : tile_up(c, 0, fx, fy, bu, bv, xu, xv, nu);
    return st;
  }
  for (int s = 0; s < sweeps; ++s) {
    int st = gs_sweep(c, 0, c->kv[KV_X][0], c->kv[KV_X][1], c->kv[KV_B][0], c->kv[KV_B][1], true);
    if (st) return st;
  }
  return DIVA_OK;
}

// compulsory FP64 values per fine-level point moved by one solver_smooth_fine(c, 1)
int solver_smooth_fine_values(const Ctx* c) {
  // tiled, per point and component pair: pre reads b_u, b_v and N_a, N_b, beta_x, beta_y
  // and the two inverse diagonals (8) and writes x_u, x_v, r_u, r_v (4); post reads x_u,
  // x_v, b_u, b_v and the same 6 coefficients (10) and writes x_u, x_v (2)
  return (c->tiled && c->nlev > 1 && sub_first_level(c) > 0) ? 24 : 10;
}

int solver_matvec_fine(Ctx* c, int reps) {
  auto K = c->kv;
  for (int r = 0; r < reps; ++r) {
    k_matvec<<<red_blocks(c->d), block2d(), 0, c->stream>>>(make_op(c, 0), K[KV_X][0], K[KV_X][1], K[KV_T][0], K[KV_T][1],
                                                            K[KV_RHAT][0], K[KV_RHAT][1], reduction(c), c->scal,
                                                            ST_NONE); c->launches++;
  }
  DIVA_LAUNCHED(c, "k_matvec");
  return DIVA_OK;
}

// one preconditioner application (V-cycle from zero) on the current Krylov residual
int solver_vcycle_fine(Ctx* c, int reps) {
  for (int r = 0; r < reps; ++r) {
    int st = precond(c, c->kv[KV_R][0], c->kv[KV_R][1], c->kv[KV_PHAT][0], c->kv[KV_PHAT][1]);
    if (st) return st;
  }
  return DIVA_OK;
}

// the one-block part of the V-cycle alone, on the arrays of its first level
int solver_subcycle(Ctx* c, int reps) {
  const int l = sub_first_level(c);
  const Level& L = c->lv[l];
  for (int r = 0; r < reps; ++r) {
    int st = vcycle(c, l, L.xu, L.xv, L.bu, L.bv, Restriction{});
    if (st) return st;
  }
  return DIVA_OK;
}

// algorithmic bytes of one V-cycle (FP64, compulsory traffic per point and level):
// each sweep 10 values, the residual 8, the transfers 6, weighted by the level's points
double solver_vcycle_bytes(const Ctx* c) {
  double b = 0.0;
  for (int l = 0; l < c->nlev; ++l)
    b += (double)c->lv[l].d.nx * c->lv[l].d.ny * sizeof(double) * (4 * 10 + 8 + 6);
  return b;
}

// row types of the finest level (choice_ice_margin 'BC'), from the SICO masks of this solve
int solver_row_types(Ctx* c) {
  if (c->c.choice_ice_margin != DIVA_MARGIN_BC) return DIVA_OK;
  k_row_types<<<GL(0)>>>(c->d, c->I(DIVA_F_DIVA_MASK_COMBI), c->I(DIVA_F_DIVA_ISFRONT_INNER),
                         c->I(DIVA_F_DIVA_ISFRONT_OUTER), c->rtu, c->rtv); c->launches++;
  DIVA_LAUNCHED(c, "k_row_types");
  return DIVA_OK;
}

// ---- the viscosity iteration loop as one CUDA graph -------------------------------
//
// One viscosity iteration (ITER):
//   pre   : coefficients (K1 + faces; K1 also starts the iteration's counters), operator
//           set-up of all levels, x <- (u,v) and the initial residual with the nonlinear
//           one, which [relres stop rule] sets IF(solve)
//   IF(solve):
//     head  : k_ctl_lin_init sets WHILE(krylov)
//     WHILE(krylov):
//       first : V-cycle p -> phat, v = A phat, alpha, s, whose norm sets IF(second)
//               and may end the loop
//       IF(second): V-cycle s -> shat, t = A shat, omega, x and r, whose norm sets
//                   WHILE(krylov), p update
//     tail  : the solution (half step, boundary), Picard update (limits, relaxation, step
//             norm, basal stress and velocity, DIVA_err), stop test
//   the loop goes on unless the iteration converged, the residual met its tolerance, a NaN
//   appeared or the iteration budget is spent: decided by the Picard update (step-norm rule)
//   or [relres stop rule] by the post kernel, which also forms the basal stress and velocity
//   of an iteration the residual stopped
//
// The whole loop: WHILE(picard) { ITER(parity p); IF(odd) { ITER(parity 1 - p) } }.
// The viscosity is double-buffered (each iteration reads one buffer and writes the
// other), and captured kernel arguments are fixed pointers, so the body holds two
// iterations, one per buffer order; the first sets IF(odd) to its continue flag.
// Two instances are built, one per starting buffer; one launch runs a whole solve
// with no host round trip between iterations.
namespace {

struct CaptureCtx {
  Ctx* c;
  cudaStream_t s[6] = {};
  bool capturing[6] = {};
  long long l0 = 0;
  double p0 = 0.0;
  void mark() { l0 = c->launches; p0 = c->fine_passes; }
  long long dl() const { return c->launches - l0; }
  double dp() const { return c->fine_passes - p0; }
};

int add_conditional(Ctx* c, cudaStream_t s, cudaGraphConditionalHandle h, cudaGraphConditionalNodeType type,
                    cudaGraph_t* body) {
  cudaStreamCaptureStatus st;
  cudaGraph_t g = nullptr;
  const cudaGraphNode_t* deps = nullptr;
  size_t nd = 0;
  DIVA_CUDA(c, cudaStreamGetCaptureInfo(s, &st, nullptr, &g, &deps, &nd));
  if (st != cudaStreamCaptureStatusActive) return set_error(c, DIVA_CUDA_ERROR, "stream is not capturing");
  cudaGraphNodeParams p = {};
  p.type = cudaGraphNodeTypeConditional;
  p.conditional.handle = h;
  p.conditional.type = type;
  p.conditional.size = 1;
  cudaGraphNode_t node;
  DIVA_CUDA(c, cudaGraphAddNode(&node, g, deps, nd, &p));
  *body = p.conditional.phGraph_out[0];
  DIVA_CUDA(c, cudaStreamUpdateCaptureDependencies(s, &node, 1, cudaStreamSetCaptureDependencies));
  return DIVA_OK;
}

// the graph a capturing stream records into
int capture_graph(Ctx* c, cudaStream_t s, cudaGraph_t* g) {
  cudaStreamCaptureStatus st;
  DIVA_CUDA(c, cudaStreamGetCaptureInfo(s, &st, nullptr, g, nullptr, nullptr));
  if (st != cudaStreamCaptureStatusActive) return set_error(c, DIVA_CUDA_ERROR, "stream is not capturing");
  return DIVA_OK;
}

// One viscosity iteration recorded into the graph that stream `top` is capturing; its
// conditional bodies use cc.s[3..5].  `count`: record the launches and passes of its parts.
int capture_iteration(Ctx* c, CaptureCtx& cc, cudaStream_t top, bool diva, PicardGraphs& G, bool count,
                      cudaGraphConditionalHandle h_a, cudaGraphConditionalHandle h_b, int has_b) {
  const diva_config_t& C = c->c;
  const bool relmode = C.picard_stop == DIVA_STOP_RELRES;
  auto U_ = [&](int k) { return c->kv[k][0]; };
  auto V_ = [&](int k) { return c->kv[k][1]; };
  double* u = c->D(diva ? DIVA_F_U_VAV_CX : DIVA_F_U_SSA_CX);
  double* v = c->D(diva ? DIVA_F_V_VAV_CY : DIVA_F_V_SSA_CY);
  int st;
  cudaGraph_t graph;
  if ((st = capture_graph(c, top, &graph))) return st;
  cudaGraphConditionalHandle h_solve;
  DIVA_CUDA(c, cudaGraphConditionalHandleCreate(&h_solve, graph, 1, cudaGraphCondAssignDefault));
  c->stream = top;
  const IterEnd end{1, relmode ? 0 : 1, C.DIVA_visc_it_nit, has_b, C.DIVA_visc_it_norm_dUV_tol, h_a, h_b};
  // ---- pre
  cc.mark();
  if ((st = launch_diva_coefficients(c, u, v, diva, K1_LOOP, true))) return st;   // swaps the viscosity buffers
  if ((st = solver_setup(c, 1))) return st;
  launch_init_residual(c, u, v, relmode ? 1 : 0,
                       RelresTest{relmode ? 1 : 0, C.picard_stall_its, C.picard_relres_tol, h_solve});
  DIVA_LAUNCHED(c, "graph pre");
  if (count) { G.n_pre = cc.dl(); G.p_pre = cc.dp(); }
  // ---- IF(solve)
  cudaGraph_t body_solve;
  if ((st = add_conditional(c, top, h_solve, cudaGraphCondTypeIf, &body_solve))) return st;
  cudaGraphConditionalHandle h_while;
  DIVA_CUDA(c, cudaGraphConditionalHandleCreate(&h_while, body_solve, 0, cudaGraphCondAssignDefault));
  DIVA_CUDA(c, cudaStreamBeginCaptureToGraph(cc.s[3], body_solve, nullptr, nullptr, 0,
                                             cudaStreamCaptureModeThreadLocal));
  cc.capturing[3] = true;
  c->stream = cc.s[3];
  cc.mark();
  k_ctl_lin_init<<<1, 1, 0, c->stream>>>(c->scal, h_while, relmode && C.lin_adaptive, C.lin_rtol, C.lin_maxit); c->launches++;
  DIVA_LAUNCHED(c, "graph head");
  if (count) { G.n_head = cc.dl(); G.p_head = cc.dp(); }
  // ---- WHILE(krylov)
  cudaGraph_t body_while;
  if ((st = add_conditional(c, cc.s[3], h_while, cudaGraphCondTypeWhile, &body_while))) return st;
  cudaGraphConditionalHandle h_half;
  DIVA_CUDA(c, cudaGraphConditionalHandleCreate(&h_half, body_while, 1, cudaGraphCondAssignDefault));
  DIVA_CUDA(c, cudaStreamBeginCaptureToGraph(cc.s[4], body_while, nullptr, nullptr, 0,
                                             cudaStreamCaptureModeThreadLocal));
  cc.capturing[4] = true;
  c->stream = cc.s[4];
  cc.mark();
  if ((st = precond(c, U_(KV_P), V_(KV_P), U_(KV_PHAT), V_(KV_PHAT)))) return st;
  launch_first_half(c, LoopHandles{1, h_while, h_half});
  DIVA_LAUNCHED(c, "graph first half");
  if (count) { G.n_first = cc.dl(); G.p_first = cc.dp(); }
  // ---- IF(second half)
  cudaGraph_t body_half;
  if ((st = add_conditional(c, cc.s[4], h_half, cudaGraphCondTypeIf, &body_half))) return st;
  DIVA_CUDA(c, cudaStreamBeginCaptureToGraph(cc.s[5], body_half, nullptr, nullptr, 0,
                                             cudaStreamCaptureModeThreadLocal));
  cc.capturing[5] = true;
  c->stream = cc.s[5];
  cc.mark();
  if ((st = precond(c, U_(KV_S), V_(KV_S), U_(KV_SHAT), V_(KV_SHAT)))) return st;
  launch_second_half(c, LoopHandles{1, h_while, h_while});
  DIVA_LAUNCHED(c, "graph second half");
  if (count) { G.n_second = cc.dl(); G.p_second = cc.dp(); }
  DIVA_CUDA(c, cudaStreamEndCapture(cc.s[5], &body_half));
  cc.capturing[5] = false;
  DIVA_CUDA(c, cudaStreamEndCapture(cc.s[4], &body_while));
  cc.capturing[4] = false;
  // ---- tail
  c->stream = cc.s[3];
  cc.mark();
  launch_finish_x(c, -1);
  DIVA_LAUNCHED(c, "graph tail");
  if (C.picard_anderson_m > 0 && (st = launch_anderson_prepare(c, u, v, U_(KV_XF), V_(KV_XF)))) return st;
  if ((st = launch_picard_update(c, u, v, U_(KV_XF), V_(KV_XF), diva, -1, &end))) return st;
  if (count) { G.n_tail = cc.dl(); G.p_tail = cc.dp(); }
  DIVA_CUDA(c, cudaStreamEndCapture(cc.s[3], &body_solve));
  cc.capturing[3] = false;
  // ---- post
  c->stream = top;
  cc.mark();
  if (relmode && (st = launch_relres_end(c, diva, end))) return st;
  if (count) G.n_post = cc.dl();
  return DIVA_OK;
}

// The whole viscosity loop of one context, WHILE(picard) { ITER(parity); IF(odd) { ITER(1 -
// parity) } }, appended to `graph` as a root node (no dependencies): on its own the graph of
// build_one, several of them side by side the graph of a batch (solver_build_batch_graph).
int capture_loop(Ctx* c, CaptureCtx& cc, bool diva, PicardGraphs& G, int parity, cudaGraph_t graph, bool count) {
  cudaGraphConditionalHandle h_pic;
  DIVA_CUDA(c, cudaGraphConditionalHandleCreate(&h_pic, graph, 1, cudaGraphCondAssignDefault));
  DIVA_CUDA(c, cudaStreamBeginCaptureToGraph(cc.s[0], graph, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
  cc.capturing[0] = true;
  G.visc_buf[parity] = c->f[DIVA_F_VISC_EFF_3D_A];
  int st;
  cudaGraph_t body_pic;
  if ((st = add_conditional(c, cc.s[0], h_pic, cudaGraphCondTypeWhile, &body_pic))) return st;
  DIVA_CUDA(c, cudaStreamBeginCaptureToGraph(cc.s[1], body_pic, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
  cc.capturing[1] = true;
  cudaGraphConditionalHandle h_odd;
  DIVA_CUDA(c, cudaGraphConditionalHandleCreate(&h_odd, body_pic, 0, cudaGraphCondAssignDefault));
  // the first iteration of the pair (its buffer order is this graph's parity)
  if ((st = capture_iteration(c, cc, cc.s[1], diva, G, count, h_pic, h_odd, 1))) return st;
  cudaGraph_t body_odd;
  if ((st = add_conditional(c, cc.s[1], h_odd, cudaGraphCondTypeIf, &body_odd))) return st;
  DIVA_CUDA(c, cudaStreamBeginCaptureToGraph(cc.s[2], body_odd, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
  cc.capturing[2] = true;
  if ((st = capture_iteration(c, cc, cc.s[2], diva, G, false, h_pic, h_pic, 0))) return st;
  DIVA_CUDA(c, cudaStreamEndCapture(cc.s[2], &body_odd));
  cc.capturing[2] = false;
  DIVA_CUDA(c, cudaStreamEndCapture(cc.s[1], &body_pic));
  cc.capturing[1] = false;
  cudaGraph_t top = nullptr;
  DIVA_CUDA(c, cudaStreamEndCapture(cc.s[0], &top));
  cc.capturing[0] = false;
  return DIVA_OK;
}

// the loop graph starting from the viscosity buffer `parity`
int build_one(Ctx* c, CaptureCtx& cc, bool diva, PicardGraphs& G, int parity) {
  cudaGraph_t graph;
  DIVA_CUDA(c, cudaGraphCreate(&graph, 0));
  int st = capture_loop(c, cc, diva, G, parity, graph, parity == 0);
  if (st) {
    cudaGraphDestroy(graph);
    return st;
  }
  cudaGraphExec_t exec = nullptr;
  const cudaError_t e = cudaGraphInstantiate(&exec, graph, 0);
  cudaGraphDestroy(graph);
  DIVA_CUDA(c, e);
  G.exec[parity] = exec;
  return DIVA_OK;
}

// end every capture a failed build left open, and forget the error it left behind
void close_captures(CaptureCtx& cc) {
  for (int q = 5; q >= 0; --q) {
    if (cc.capturing[q]) {
      cudaGraph_t junk = nullptr;
      cudaStreamEndCapture(cc.s[q], &junk);
      if (junk) cudaGraphDestroy(junk);
      cc.capturing[q] = false;
    }
  }
  cudaGetLastError();
}

}  // namespace

int solver_tile_edges(const Ctx* c, int32_t* edges, int n) {
  const int first = sub_first_level(c);
  for (int l = 0; l < n; ++l)
    edges[l] = (l < c->nlev && c->tiled && c->nlev > 1 && l < first) ? tile_edge(c, l) : 0;
  return c->nlev;
}

int solver_strip_rows(const Ctx* c, int32_t* rows, int n) {
  const int first = sub_first_level(c);
  for (int l = 0; l < n; ++l) {
    const bool strips = l < c->nlev && c->tiled && c->nlev > 1 && l < first && level_streamed(c, l);
    rows[l] = strips ? wave_shape(c->lv[l].d.ny, c->lv[l].d.nx).rows : 0;
  }
  return c->nlev;
}

void solver_destroy_graphs(Ctx* c) {
  for (auto& G : c->graphs) {
    for (auto& e : G.exec)
      if (e) cudaGraphExecDestroy(e), e = nullptr;
    G.valid = false;
  }
}

int solver_build_picard_graphs(Ctx* c, bool diva) {
  PicardGraphs& G = c->graphs[diva ? 1 : 0];
  if (G.valid) return DIVA_OK;
  CaptureCtx cc;
  cc.c = c;
  cudaStream_t user = c->stream;
  const long long launches0 = c->launches;
  const double passes0 = c->fine_passes;
  const long mg0 = c->mg_cycles;
  void* visc0 = c->f[DIVA_F_VISC_EFF_3D_A];
  double* prev0 = c->visc_prev;
  int st = DIVA_OK;
  for (int q = 0; q < 6 && !st; ++q)
    if (cudaStreamCreateWithFlags(&cc.s[q], cudaStreamNonBlocking) != cudaSuccess) st = DIVA_CUDA_ERROR;
  // parity 0 starts from the current buffer, parity 1 from the other; each graph
  // captures two iterations, which swap the viscosity buffers twice
  for (int parity = 0; parity < 2 && !st; ++parity) {
    if (parity == 1) std::swap(c->f[DIVA_F_VISC_EFF_3D_A], *reinterpret_cast<void**>(&c->visc_prev));
    st = build_one(c, cc, diva, G, parity);
  }
  close_captures(cc);   // and clear any capture error so the host path can proceed
  for (int q = 0; q < 6; ++q)
    if (cc.s[q]) cudaStreamDestroy(cc.s[q]);
  c->stream = user;
  c->launches = launches0;
  c->fine_passes = passes0;
  c->mg_cycles = mg0;
  c->f[DIVA_F_VISC_EFF_3D_A] = visc0;   // the captures swap these without running anything
  c->visc_prev = prev0;
  if (st) {
    for (auto& e : G.exec)
      if (e) cudaGraphExecDestroy(e), e = nullptr;
    return st;
  }
  G.valid = true;
  return DIVA_OK;
}

// One graph holding the viscosity loops of n contexts side by side (a batch, diva_batch_create):
// each member's loop is captured as it stands now (its viscosity buffer order, its
// configuration) into one parent graph, instantiated once.  bufs[k] receives the buffer
// member k's loop starts from.  Every member's own loop graphs must exist already (their
// launch and pass counts account for the batch's iterations).
int solver_build_batch_graph(Ctx* const* cs, int n, cudaGraphExec_t* exec, void** bufs) {
  Ctx* c0 = cs[0];
  *exec = nullptr;
  cudaGraph_t parent = nullptr;
  DIVA_CUDA(c0, cudaGraphCreate(&parent, 0));
  CaptureCtx cc;
  int st = DIVA_OK;
  for (int q = 0; q < 6 && !st; ++q)
    if (cudaStreamCreateWithFlags(&cc.s[q], cudaStreamNonBlocking) != cudaSuccess) st = DIVA_CUDA_ERROR;
  for (int k = 0; k < n && !st; ++k) {
    Ctx* c = cs[k];
    cc.c = c;
    PicardGraphs scratch;   // the loop's counts are the member's own graphs'
    cudaStream_t user = c->stream;
    const long long launches0 = c->launches;
    const double passes0 = c->fine_passes;
    const long mg0 = c->mg_cycles;
    void* visc0 = c->f[DIVA_F_VISC_EFF_3D_A];
    double* prev0 = c->visc_prev;
    bufs[k] = visc0;
    st = capture_loop(c, cc, true, scratch, 0, parent, false);
    c->stream = user;
    c->launches = launches0;
    c->fine_passes = passes0;
    c->mg_cycles = mg0;
    c->f[DIVA_F_VISC_EFF_3D_A] = visc0;   // the capture swaps these without running anything
    c->visc_prev = prev0;
    if (st) set_error(c0, st, "batch graph: capture of member " + std::to_string(k) + " failed: " + c->err);
  }
  close_captures(cc);
  for (int q = 0; q < 6; ++q)
    if (cc.s[q]) cudaStreamDestroy(cc.s[q]);
  if (!st && cudaGraphInstantiate(exec, parent, 0) != cudaSuccess) {
    *exec = nullptr;
    cudaGetLastError();
    st = set_error(c0, DIVA_CUDA_ERROR, "batch graph: instantiation failed");
  }
  cudaGraphDestroy(parent);
  return st;
}

}  // namespace diva
