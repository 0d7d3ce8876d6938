// picard.cu -- the per-iteration physics of solve_DIVA / solve_SSA and the
// velocity fields computed after the viscosity iteration.
//
//   K1 k_column_prep, k_layer_viscosity, k_column_integrals (+ k_shear_rates once per solve)
//                             calc_vertical_shear_strain_rates   ice_velocity_module.f90:664-721
//                             calc_effective_viscosity (a-grid)   :722-818
//                             calc_sliding_term_beta + laws       :900-959, basal_conditions_and_sliding_module.f90:908-1236
//                             calc_F_integral(n=2)                :960-1013
//                             calc_beta_eff (a-grid)              :1014-1061
//      k_face_coefficients    N_b (:820-874), N_cx/N_cy (:876-880), beta_eff on cx/cy (:1063-1076)
//   K4 k_picard_update        apply_velocity_limits :1432-1498, relax :1499-1529,
//                             calc_visc_iter_UV_resid :1530-1601 (block partials),
//                             estimate_visc_iter_UV_errors :1602-1652,
//                             calc_basal_stress :1087-1120, calc_basal_velocities :1121-1199
//   K5 k_f1 / k_u3d           calc_3D_horizontal_velocities_DIVA  :1200-1298
//   K6 k_faces_prelude / k_secondary
//                             calc_secondary_velocities :377-533, calc_3D_vertical_velocities :534-661,
//                             map_velocity_from_c*_to_a_* :2592-2811
//   K7 k_sia                  solve_SIA :36-105
//
// One thread owns one a-grid column (j,i) and, with it, the cx face (j,i) east
// of it and the cy face (j,i) north of it.  Column loops run over the zeta
// layers, each a coalesced plane.
#include <algorithm>
#include <cmath>
#include <math_constants.h>
#include "ctx.hpp"

namespace diva {
namespace {

struct CoefArgs {
  Dims d;
  Zeta zt;
  // config
  int diva, bc_margin, sliding, gl_subgrid, basal_freezing, prescribed_tauc, n_is_3, crossterms;
  double n_flow, eps0, visc_min, beta_max, delta_v, wm, q_plastic, u_thr, zi_ut, zi_p, dT_freeze, Fmin;
  // inputs
  const double *u, *v, *visc_prev, *taub_cx, *taub_cy, *Hi, *afac;
  const int *mask_ice, *mask_ocean;
  const double *beta_sq, *phi_fric, *alpha_sq, *Neff, *Ti, *Tpmp;
  // outputs
  double *dudz, *dvdz, *visc, *visc_int, *Na, *beta, *F2, *beta_eff, *tauc;
  // per-column scratch between the three launches
  double* col_eps;
  int* col_flags;
  // the basal stress each column's shear read, kept (keep_seen) so that the shear strain
  // rates of the viscosity loop's last iteration can be written after the loop
  int keep_seen;
  double *taub_seen_cx, *taub_seen_cy;
  double* sc;   // device scalars of a graph-launched iteration that starts here, else null
};

// strain rates of the depth-averaged velocity on the a-grid,
// ddx_cx_to_a / ddy_cx_to_a / ddx_cy_to_a / ddy_cy_to_a (derivatives_and_grids_module.f90:755-939)
__device__ __forceinline__ double ddx_cx_to_a(const Dims& d, const double* u, int j, int i) {
  const int ii = i == 0 ? 1 : (i == d.nx - 1 ? d.nx - 2 : i);
  return (u[d.at(j, ii)] - u[d.at(j, ii - 1)]) / d.dx;
}
__device__ __forceinline__ double ddy_cy_to_a(const Dims& d, const double* v, int j, int i) {
  const int jj = j == 0 ? 1 : (j == d.ny - 1 ? d.ny - 2 : j);
  return (v[d.at(jj, i)] - v[d.at(jj - 1, i)]) / d.dx;
}
__device__ __forceinline__ double ddy_cx_to_a(const Dims& d, const double* u, int j, int i) {
  const int nx = d.nx, ny = d.ny;
  const double dx = d.dx;
  auto U = [&](int jj, int ii) { return u[d.at(jj, ii)]; };
  if (i > 0 && i < nx - 1) {
    if (j > 0 && j < ny - 1) return (U(j + 1, i - 1) + U(j + 1, i) - U(j - 1, i - 1) - U(j - 1, i)) / (4.0 * dx);
    if (j == 0) return (U(1, i - 1) + U(1, i) - U(0, i - 1) - U(0, i)) / (4.0 * dx);
    return (U(ny - 1, i - 1) + U(ny - 1, i) - U(ny - 2, i - 1) - U(ny - 2, i)) / (4.0 * dx);
  }
  const int ic = (i == 0) ? 0 : nx - 2;
  if (j > 0 && j < ny - 1) return (U(j + 1, ic) - U(j - 1, ic)) / (2.0 * dx);
  if (j == 0) return (U(1, ic) - U(0, ic)) / dx;
  return (U(ny - 1, ic) - U(ny - 2, ic)) / dx;
}
__device__ __forceinline__ double ddx_cy_to_a(const Dims& d, const double* v, int j, int i) {
  const int nx = d.nx, ny = d.ny;
  const double dx = d.dx;
  auto V = [&](int jj, int ii) { return v[d.at(jj, ii)]; };
  if (j > 0 && j < ny - 1) {
    if (i > 0 && i < nx - 1) return (V(j - 1, i + 1) + V(j, i + 1) - V(j - 1, i - 1) - V(j, i - 1)) / (4.0 * dx);
    if (i == 0) return (V(j - 1, 1) + V(j, 1) - V(j - 1, 0) - V(j, 0)) / (4.0 * dx);
    return (V(j - 1, nx - 1) + V(j, nx - 1) - V(j - 1, nx - 2) - V(j, nx - 2)) / (4.0 * dx);
  }
  const int jc = (j == 0) ? 0 : ny - 2;
  if (i > 0 && i < nx - 1) return (V(jc, i + 1) - V(jc, i - 1)) / (2.0 * dx);
  if (i == 0) return (V(jc, 1) - V(jc, 0)) / dx;
  return (V(jc, nx - 1) - V(jc, nx - 2)) / dx;
}

__device__ __forceinline__ double sliding_beta(const CoefArgs& a, long long q, double ua, double va) {
  const double uabs = sqrt(a.delta_v * a.delta_v + ua * ua + va * va);
  switch (a.sliding) {
    case DIVA_SLIDING_NONE: return 0.0;
    case DIVA_SLIDING_WEERTMAN: return a.beta_sq[q] * pow(uabs, 1.0 / a.wm - 1.0);
    case DIVA_SLIDING_COULOMB: {
      double tc = a.prescribed_tauc ? a.tauc[q] : tan((kPi / 180.0) * a.phi_fric[q]) * a.Neff[q];
      if (!a.prescribed_tauc) a.tauc[q] = tc;
      return tc / uabs;
    }
    case DIVA_SLIDING_COULOMB_REGULARISED: {
      const double tc = tan((kPi / 180.0) * a.phi_fric[q]) * a.Neff[q];
      a.tauc[q] = tc;
      return tc * pow(uabs, a.q_plastic - 1.0) / pow(a.u_thr, a.q_plastic);
    }
    case DIVA_SLIDING_TSAI2015:
      return min_ref(a.alpha_sq[q] * a.Neff[q], a.beta_sq[q] * pow(uabs, 1.0 / a.wm)) * pow(uabs, -1.0);
    case DIVA_SLIDING_SCHOOF2005: {
      const double a2 = a.alpha_sq[q], b2 = a.beta_sq[q], m = a.wm;
      return ((b2 * pow(uabs, 1.0 / m) * a2 * a.Neff[q]) / (pow(pow(b2, m) * uabs + pow(a2 * a.Neff[q], m), 1.0 / m))) *
             pow(uabs, -1.0);
    }
    case DIVA_SLIDING_ZOET_IVERSON:
      return a.Neff[q] * tan((kPi / 180.0) * a.phi_fric[q]) * (pow(uabs, 1.0 / a.zi_p - 1.0)) *
             (pow(uabs + a.zi_ut, -1.0 / a.zi_p));
  }
  return CUDART_NAN;
}

// Block shape of the layer-parallel kernels: a warp over 32 rows, 8 grid columns.
constexpr int kColLanes = 32, kColRows = 8;

// Per-column decisions of the layer step, packed by k_column_prep (and kept for k_shear_rates):
//   bits 0-3   the E, W, N, S shear face carries ice (FACE_*)
//   bits 4-11  per face, which side the staggered viscosity takes (calc_staggered_margin
//              :1300-1319): 0 the mean of both, 1 the first (west/south) side, 2 the second
//   bits 12-15 the same choice for the column's own x and y staggering of du/dz, dv/dz,
//              including the first/last grid column and row, which take one face only
//   bit 16     no viscosity in this column (BC margins outside the ice)
enum { FACE_E = 1, FACE_W = 2, FACE_N = 4, FACE_S = 8, COL_SKIP = 1 << 16 };
constexpr int kModeShift = 4, kStagXShift = 12, kStagYShift = 14;

__device__ __forceinline__ int margin_mode(double H0, double H1) {
  if (H0 > 0.0 && H1 == 0.0) return 1;
  if (H0 == 0.0 && H1 > 0.0) return 2;
  return 0;
}
// K1 in three launches.  (a) k_column_prep, one thread per column: the strain rates
// of the depth-averaged flow and which of the column's four shear faces have ice.
// (b) k_layer_viscosity, one thread per column and one or three layers, a warp over 32
// neighbouring rows j of one grid column i: the shear of the column's own east and
// north faces, the west face, and the south face as the north face of the lane below
// (shuffle), then the viscosity of the layer.  (c) k_column_integrals, one thread per
// column: the vertical integrals in layer order (as the sequential quadrature does), N_a,
// the sliding law, F2 and beta_eff.  The middle step is layer-parallel (15 x the threads
// of a column kernel): a single column kernel walking the layers, measured, took 104 us
// per iteration on the 321 x 561 ice cap against 75 us for the three launches, whose extra
// read of the viscosity is cheaper than the lost parallelism.  The shear strain rates
// du/dz, dv/dz (:664-721) are written by the layer step only with WRITE_SHEAR; inside the
// viscosity loop (K1_LOOP) k_column_prep keeps the basal stress it saw instead, and
// k_shear_rates writes the last iteration's shear once after the loop.
__global__ void __launch_bounds__(256) k_column_prep(CoefArgs a) {
  const Dims d = a.d;
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
  if (j == 0 && i == 0 && a.sc) {   // the iteration's counters (nothing else here reads them)
    a.sc[SC_PIC_IT] += 1.0;
    a.sc[SC_EXIT_RELRES] = a.sc[SC_LIN_IT] = a.sc[SC_LIN_FULL] = a.sc[SC_SOLVED] = a.sc[SC_CONVERGED] = 0.0;
  }
  if (j >= d.ny || i >= d.nx) return;
  const int nx = d.nx, ny = d.ny;
  const long long q = d.at(j, i);
  const int* __restrict__ mask = a.mask_ice;
  const double* __restrict__ Hi = a.Hi;
  const bool ice = mask[q] == 1;
  const bool skip_visc = a.bc_margin && !ice;  // BC margins: no viscosity outside the ice (:759-764)
  // strain rates of the depth-averaged flow (calc_effective_viscosity :751-754)
  double eps_h = 0.0;
  if (!skip_visc) {
    const double du_dx = ddx_cx_to_a(d, a.u, j, i), dv_dy = ddy_cy_to_a(d, a.v, j, i);
    const double du_dy = ddy_cx_to_a(d, a.u, j, i), dv_dx = ddx_cy_to_a(d, a.v, j, i);
    eps_h = du_dx * du_dx + dv_dy * dv_dy + du_dx * dv_dy + 0.25 * ((du_dy + dv_dx) * (du_dy + dv_dx));
  }
  const double H = Hi[q];
  int flags = skip_visc ? COL_SKIP : 0;
  auto face = [&](int bit, int f, long long p0, long long p1) {
    // a face carries shear if either side has ice (calc_vertical_shear_strain_rates :685-695)
    if (a.diva && !(mask[p0] == 0 && mask[p1] == 0)) flags |= bit;
    flags |= margin_mode(Hi[p0], Hi[p1]) << (kModeShift + 2 * f);
  };
  if (i < nx - 1) face(FACE_E, 0, q, d.at(j, i + 1));
  if (i > 0) face(FACE_W, 1, d.at(j, i - 1), q);
  if (j < ny - 1) face(FACE_N, 2, q, d.at(j + 1, i));
  if (j > 0) face(FACE_S, 3, d.at(j - 1, i), q);
  // a-grid staggering of the face values: first column/row the east/north face alone (2),
  // last column/row the west/south face alone (1), else the margin rule
  const int mx = i == 0 ? 2 : (i == nx - 1 ? 1 : margin_mode(Hi[d.at(j, i - 1)], H));
  const int my = j == 0 ? 2 : (j == ny - 1 ? 1 : margin_mode(Hi[d.at(j - 1, i)], H));
  flags |= (mx << kStagXShift) | (my << kStagYShift);
  a.col_eps[q] = eps_h;
  a.col_flags[q] = flags;
  if (a.keep_seen && a.diva) {   // the basal stress this iteration's shear reads (k_shear_rates)
    if (i < nx - 1) a.taub_seen_cx[q] = a.taub_cx[q];
    if (j < ny - 1) a.taub_seen_cy[q] = a.taub_cy[q];
  }
}

// The layer step's arithmetic type R: double, or float for precision 'mixed' (the
// viscosity of the linearisation in FP32: face shears, strain rate, the rate factor's
// power and the viscosity bound; inputs and the stored viscosity stay FP64 fields).
// (calc_staggered_margin with the side choice made beforehand: same values as stag_margin)
template <class R> __device__ __forceinline__ R stag_mode_t(int mode, R v0, R v1) {
  return mode == 1 ? v0 : (mode == 2 ? v1 : R(0.5) * (v0 + v1));
}
template <class R> __device__ __forceinline__ R max_ref_t(R a, R b) { return (b > a || a != a) ? b : a; }
__device__ __forceinline__ double rcbrt_t(double x) { return rcbrt(x); }
__device__ __forceinline__ float rcbrt_t(float x) { return rcbrtf(x); }
__device__ __forceinline__ double pow_t(double x, double y) { return pow(x, y); }
__device__ __forceinline__ float pow_t(float x, float y) { return powf(x, y); }

// A thread takes L layers of its column, whose loads are in flight together and share the
// column's flags and basal stress.  All of K1 in FP64, 15 layers, one layer a thread against three:
// 23.6 / 25.6 us on 129 x 17, 25.7 / 26.7 on 257 x 33, 26.7 / 28.2 on 81 x 141, 28.7 / 30.8 on
// 115 x 201, 32.8 / 32.9 on 161 x 281, 38.0 / 36.9 on 201 x 351, 77.0 / 72.8 on 321 x 561, 198 / 175 on
// 533 x 933.  Three where a GPU of 2048 threads per SM is full with them, one below: there a
// thread's layers come one after the other while SMs are idle (two are between the others; five
// at 321 x 561, 1501 x 1501 and 129 x 17 84.9, 804 and 27.8 us: too few warps for their registers).
constexpr int kViscLayers = 3;
inline int visc_layers(const Dims& d) {
  return (long long)d.nx * d.ny * ((d.nz + kViscLayers - 1) / kViscLayers) >= 2048LL * kSMs ? kViscLayers : 1;
}
template <bool WRITE_SHEAR, class R, int L>
__global__ void __launch_bounds__(kColLanes * kColRows) k_layer_viscosity(CoefArgs a) {
  const Dims d = a.d;
  const int lane = threadIdx.x, y = threadIdx.y;
  // the layers are the fastest grid index: blocks running together share their columns'
  // 2D inputs in L1/L2 instead of streaming them once per layer
  const int k0 = blockIdx.x * L, j = blockIdx.y * kColLanes + lane, i = blockIdx.z * kColRows + y;
  const bool row = i < d.nx;   // whole warps: i is uniform across a warp; idle warps stay for the barrier
  const bool col = row && j < d.ny;   // lanes past the last row stay for the shuffle
  const int nx = d.nx, ny = d.ny, ld = d.ld;
  const int q = (row ? i : nx - 1) * ld + (j < ny ? j : ny - 1);   // plane index (planes hold < 2^31 points)
  const int flags = a.col_flags[q];
  const bool has_e = col && i < nx - 1, has_w = col && i > 0, has_n = col && j < ny - 1, has_s = col && j > 0;
  const bool on_e = has_e && (flags & FACE_E), on_n = has_n && (flags & FACE_N);
  const bool on_w = has_w && (flags & FACE_W), on_s = has_s && (flags & FACE_S);
  const bool skip = flags & COL_SKIP;
  auto mode = [&](int f) { return (flags >> (kModeShift + 2 * f)) & 3; };
  auto shear = [](double tb, double v0, double v1, int m, R zk) { return ((R)tb / stag_mode_t<R>(m, (R)v0, (R)v1)) * zk; };
  auto layer = [&](int e) { return k0 + e < d.nz ? k0 + e : d.nz - 1; };   // (the last again where there are fewer)
  const double eps = skip ? 0.0 : a.col_eps[q];
  double af[L];
#pragma unroll
  for (int e = 0; e < L; ++e) af[e] = a.afac[layer(e) * d.plane + q];
  // the west face of column i is the east face of column i-1: the warp below in the block
  // computed it (the same operands, so the same value), the block's first warp computes it;
  // the south face of row j is the north face of row j-1, the lane below's
  __shared__ R east[L][kColRows][kColLanes];
  R dudz_e[L] = {}, dvdz_n[L] = {}, dvdz_s[L] = {}, dudz_w[L] = {};
  if (a.diva) {
    const double te = on_e ? a.taub_cx[q] : 0.0, tn = on_n ? a.taub_cy[q] : 0.0;
    const bool edge_w = y == 0 && on_w, edge_s = lane == 0 && on_s;
    const double tw = edge_w ? a.taub_cx[q - ld] : 0.0, ts = edge_s ? a.taub_cy[q - 1] : 0.0;
    double vq[L], ve[L], vn[L], vw[L], vs[L];
#pragma unroll
    for (int e = 0; e < L; ++e) {
      const double* __restrict__ vp = a.visc_prev + layer(e) * d.plane;
      vq[e] = vp[q];
      ve[e] = on_e ? vp[q + ld] : 0.0;
      vn[e] = on_n ? vp[q + 1] : 0.0;
      vw[e] = edge_w ? vp[q - ld] : 0.0;
      vs[e] = edge_s ? vp[q - 1] : 0.0;
    }
#pragma unroll
    for (int e = 0; e < L; ++e) {
      const R zk = (R)a.zt.z[layer(e)];
      if (on_e) dudz_e[e] = shear(te, vq[e], ve[e], mode(0), zk);
      if (on_n) dvdz_n[e] = shear(tn, vq[e], vn[e], mode(2), zk);
      if (edge_w) dudz_w[e] = shear(tw, vw[e], vq[e], mode(1), zk);
      if (edge_s) dvdz_s[e] = shear(ts, vs[e], vq[e], mode(3), zk);
      east[e][y][lane] = dudz_e[e];
      if (WRITE_SHEAR && k0 + e < d.nz) {
        const long long o = (k0 + e) * d.plane + q;
        if (has_e) a.dudz[o] = (double)dudz_e[e];
        if (has_n) a.dvdz[o] = (double)dvdz_n[e];
      }
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < L; ++e) {
      const R below = __shfl_up_sync(0xffffffffu, dvdz_n[e], 1);
      if (lane > 0) dvdz_s[e] = below;
      if (y > 0 && on_w) dudz_w[e] = east[e][y - 1][lane];
    }
  }
  if (!col) return;
  const int mx = (flags >> kStagXShift) & 3, my = (flags >> kStagYShift) & 3;
  const R flow = a.n_is_3 ? R(0) : (R)((1.0 - a.n_flow) / (2.0 * a.n_flow));
#pragma unroll
  for (int e = 0; e < L; ++e) {
    if (k0 + e >= d.nz) break;
    const long long off = (k0 + e) * d.plane;
    R eta = R(0);
    if (!skip) {
      R du_dz_a, dv_dz_a;
      if (a.diva) {
        du_dz_a = stag_mode_t<R>(mx, dudz_w[e], dudz_e[e]);
        dv_dz_a = stag_mode_t<R>(my, dvdz_s[e], dvdz_n[e]);
      } else {
        // solve_SSA calls calc_effective_viscosity without refreshing du/dz: use the stored fields
        const double* dudz = a.dudz + off;
        const double* dvdz = a.dvdz + off;
        du_dz_a = stag_mode_t<R>(mx, (R)(i > 0 ? dudz[q - ld] : 0.0), (R)(i < nx - 1 ? dudz[q] : 0.0));
        dv_dz_a = stag_mode_t<R>(my, (R)(j > 0 ? dvdz[q - 1] : 0.0), (R)(j < ny - 1 ? dvdz[q] : 0.0));
      }
      const R eps_sq = (R)eps + R(0.25) * (du_dz_a * du_dz_a + dv_dz_a * dv_dz_a) + (R)a.eps0;
      const R pe = a.n_is_3 ? rcbrt_t(eps_sq) : pow_t(eps_sq, flow);
      eta = max_ref_t<R>((R)af[e] * pe, (R)a.visc_min);   // NaN (first cold iteration) -> visc_min
    }
    a.visc[off + q] = (double)eta;
  }
}

// NZ > 0: the layer count known at compile time (the default 15 layers), so the loop is
// unrolled and every layer's load is in flight at once; NZ = 0: any layer count.
template <int NZ, class R>
__global__ void __launch_bounds__(256) k_column_integrals(CoefArgs a) {
  const Dims d = a.d;
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
  if (j >= d.ny || i >= d.nx) return;
  const int nx = d.nx, ny = d.ny, nz = NZ > 0 ? NZ : d.nz;
  const long long q = d.at(j, i);
  const double H = a.Hi[q];
  const bool ice = a.mask_ice[q] == 1;
  const bool skip_visc = a.bc_margin && !ice;
  const double* __restrict__ visc = a.visc;
  // every load ahead of the sliding law's arithmetic and of the stores
  double etas[NZ > 0 ? NZ : 1];
#pragma unroll
  for (int k = 0; k < NZ; ++k) etas[k] = visc[(long long)k * d.plane + q];
  bool frozen = false;
  if (a.diva && a.basal_freezing) {
    const long long ob = (long long)(nz - 1) * d.plane + q;
    frozen = a.Tpmp[ob] - a.Ti[ob] > a.dT_freeze;
  }
  // sliding (calc_sliding_term_beta :924-951)
  double ua, va;
  if (i == 0) ua = a.u[d.at(j, 0)];
  else if (i == nx - 1) ua = a.u[d.at(j, nx - 2)];
  else ua = (a.u[d.at(j, i - 1)] + a.u[q]) / 2.0;
  if (j == 0) va = a.v[d.at(0, i)];
  else if (j == ny - 1) va = a.v[d.at(ny - 2, i)];
  else va = (a.v[d.at(j - 1, i)] + a.v[q]) / 2.0;
  double beta = min_ref(sliding_beta(a, q, ua, va), a.beta_max);
  if (!a.gl_subgrid && a.mask_ocean[q] == 1) beta = 0.0;
  double vint = 0.0, fint = 0.0, vprev = 0.0, fprev = 0.0;
#pragma unroll
  for (int k = 0; k < nz; ++k) {
    const double eta = NZ > 0 ? etas[NZ > 0 ? k : 0] : visc[(long long)k * d.plane + q];
    const double zk = a.zt.z[k];
    if (k > 0) vint = vint + 0.5 * (eta + vprev) * (zk - a.zt.z[k - 1]);
    vprev = eta;
    if (a.diva) {
      const double fk = (double)(((R)H / (R)eta) * (R)a.zt.z2[k]);
      if (k > 0) fint = fint + 0.5 * (fk + fprev) * (zk - a.zt.z[k - 1]);
      fprev = fk;
    }
  }
  if (!skip_visc) {
    a.visc_int[q] = vint;
    a.Na[q] = a.bc_margin ? vint * H : vint * max_ref(0.1, H);
  }
  a.beta[q] = beta;
  if (a.diva) {
    double F2;
    if (ice) F2 = max_ref(a.Fmin, fint);
    else F2 = a.bc_margin ? 0.0 : a.Fmin;
    a.F2[q] = F2;
    double be;
    if (a.sliding == DIVA_SLIDING_NONE) {
      be = 1.0 / F2;
    } else {
      be = frozen ? 1.0 / F2 : beta / (1.0 + beta * F2);
    }
    a.beta_eff[q] = be;
  } else {
    a.beta_eff[q] = beta;   // solve_SSA :193
  }
}


// The shear strain rates du/dz, dv/dz (calc_vertical_shear_strain_rates :664-721) of the last
// viscosity iteration, from the flags and basal stress its fused K1 kept and the viscosity
// it read: the values a K1 that writes them would have left.  Layer-parallel.
template <class R>
__global__ void __launch_bounds__(kColLanes * kColRows) k_shear_rates(CoefArgs a) {
  const Dims d = a.d;
  const int lane = threadIdx.x;
  const int k = blockIdx.x, j = blockIdx.y * kColLanes + lane, i = blockIdx.z * kColRows + threadIdx.y;
  if (i >= d.nx) return;
  const bool col = j < d.ny;
  const int nx = d.nx, ny = d.ny, ld = d.ld;
  const long long q = d.at(col ? j : ny - 1, i);
  const long long off = (long long)k * d.plane;
  const double* __restrict__ vp = a.visc_prev + off;
  const R zk = (R)a.zt.z[k];
  const int flags = a.col_flags[q];
  auto mode = [&](int f) { return (flags >> (kModeShift + 2 * f)) & 3; };
  auto shear = [&](double tb, double v0, double v1, int m) { return ((R)tb / stag_mode_t<R>(m, (R)v0, (R)v1)) * zk; };
  if (!col) return;
  if (i < nx - 1) a.dudz[off + q] = (double)((flags & FACE_E) ? shear(a.taub_seen_cx[q], vp[q], vp[q + ld], mode(0)) : R(0));
  if (j < ny - 1) a.dvdz[off + q] = (double)((flags & FACE_N) ? shear(a.taub_seen_cy[q], vp[q], vp[q + 1], mode(2)) : R(0));
}

struct FaceArgs {
  Dims d;
  int bc_margin, apply_fgrnd, crossterms;
  const double *vint, *Hb_i, *beta_eff, *fcx, *fcy, *Na;
  const int* mask_ice;
  double *visc_int_b, *Nb, *bex, *bey, *Ncx, *Ncy;
  double *lvBx, *lvBy, *lvNa, *lvNb;   // level-0 operator coefficients (Bx = beta_eff_cx * dx^2)
};

__global__ void __launch_bounds__(256) k_face_coefficients(FaceArgs a) {
  const Dims d = a.d;
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
  if (j >= d.ny || i >= d.nx) return;
  const long long q = d.at(j, i);
  const double dx2 = d.dx * d.dx;
  const bool cx = i < d.nx - 1, cy = j < d.ny - 1;
  // every load before the first store
  const long long q1 = cx ? d.at(j, i + 1) : q, q2 = cy ? d.at(j + 1, i) : q, q3 = cx && cy ? d.at(j + 1, i + 1) : q;
  const double v0 = a.vint[q], v1 = a.vint[q1], v2 = a.vint[q2], v3 = a.vint[q3], Hb = cx && cy ? a.Hb_i[q] : 0.0;
  const double e0 = a.beta_eff[q], e1 = a.beta_eff[q1], e2 = a.beta_eff[q2];
  const double n0 = a.Na[q], n1 = a.Na[q1], n2 = a.Na[q2];
  const double fx = cx && a.apply_fgrnd ? a.fcx[q] : 0.0, fy = cy && a.apply_fgrnd ? a.fcy[q] : 0.0;
  int m0 = 1, m1 = 1, m2 = 1, m3 = 1;
  if (a.bc_margin) {
    m0 = a.mask_ice[q] == 1; m1 = a.mask_ice[q1] == 1; m2 = a.mask_ice[q2] == 1; m3 = a.mask_ice[q3] == 1;
  }
  if (cx && cy) {
    // the 3D viscosity staggered to the b-grid and integrated over the column (:820-874).
    // The staggering is a fixed weighting of the four corner columns and the trapezoid rule
    // is linear, so the integral is the same weighting of the corners' integrals (equal up
    // to rounding): the 3D viscosity is not read again.
    double s;
    if (a.bc_margin) {
      const double w = (double)m0 + (double)m1 + (double)m2 + (double)m3;
      double vb = 0.0;
      if (m0) vb = vb + v0;
      if (m1) vb = vb + v1;
      if (m2) vb = vb + v2;
      if (m3) vb = vb + v3;
      s = w > 0.0 ? vb / w : 0.0;
    } else {
      s = (v0 + v1 + v2 + v3) / 4.0;
    }
    a.visc_int_b[q] = s;
    const double nb = a.bc_margin ? s * Hb : s * max_ref(0.1, Hb);
    a.Nb[q] = nb;
    a.lvNb[q] = a.crossterms ? nb : 1.0;
  }
  if (cx) {
    double b = (e0 + e1) / 2.0;
    if (a.apply_fgrnd) b = b * (fx * fx);
    a.bex[q] = b;
    if (a.crossterms) {
      a.lvBx[q] = b * dx2;
    } else {
      const double ncx = (n0 + n1) / 2.0;
      a.Ncx[q] = ncx;
      a.lvBx[q] = dx2 * b / ncx;
    }
  }
  if (cy) {
    double b = (e0 + e2) / 2.0;
    if (a.apply_fgrnd) b = b * (fy * fy);
    a.bey[q] = b;
    if (a.crossterms) {
      a.lvBy[q] = b * dx2;
    } else {
      const double ncy = (n0 + n2) / 2.0;
      a.Ncy[q] = ncy;
      a.lvBy[q] = dx2 * b / ncy;
    }
  }
  a.lvNa[q] = a.crossterms ? n0 : 1.0;
}

// 0.5 * A^(-1/n): constant over one solve, so the pow of A is taken once per solve
__global__ void k_afac(Dims d, double n_flow, const double* A, double* afac) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y, k0 = blockIdx.z * kLayers;
  if (j >= d.ny || i >= d.nx) return;
  const double p = -1.0 / n_flow;
  const long long q = d.at(j, i);
  double f[kLayers];
  LOAD_LAYERS(e, k, k0, d.nz) f[e] = A[k * d.plane + q];
  FOR_LAYERS(e, k0, d.nz) afac[(k0 + e) * d.plane + q] = 0.5 * pow(f[e], p);
}

// apply_velocity_limits (:1432-1498) of the linear solution at a cx point: |u| with v mapped
// to the cx grid (map_cy_to_cx_2D :1757-1797), scaled down to vmax
__device__ __forceinline__ double limited_u(const Dims& d, const double* xu, const double* xv, double vmax, int j,
                                            int i) {
  const int ny = d.ny;
  auto XV = [&](int jj, int ii) { return xv[d.at(jj, ii)]; };
  double vcx;
  if (j > 0 && j < ny - 1) vcx = (XV(j - 1, i) + XV(j - 1, i + 1) + XV(j, i) + XV(j, i + 1)) / 4.0;
  else if (j == 0) vcx = (XV(0, i) + XV(0, i + 1)) / 2.0;
  else vcx = (XV(ny - 2, i) + XV(ny - 2, i + 1)) / 2.0;
  double un = xu[d.at(j, i)];
  const double uabs = sqrt(un * un + vcx * vcx);
  if (uabs > vmax) un = un * vmax / uabs;
  return un;
}
// the same at a cy point, u mapped to the cy grid (map_cx_to_cy_2D :1718-1756)
__device__ __forceinline__ double limited_v(const Dims& d, const double* xu, const double* xv, double vmax, int j,
                                            int i) {
  const int nx = d.nx;
  auto XU = [&](int jj, int ii) { return xu[d.at(jj, ii)]; };
  double ucy;
  if (i > 0 && i < nx - 1) ucy = (XU(j, i - 1) + XU(j, i) + XU(j + 1, i - 1) + XU(j + 1, i)) / 4.0;
  else if (i == 0) ucy = (XU(j, 0) + XU(j + 1, 0)) / 2.0;
  else ucy = (XU(j, nx - 2) + XU(j + 1, nx - 2)) / 2.0;
  double vn = xv[d.at(j, i)];
  const double vabs = sqrt(ucy * ucy + vn * vn);
  if (vabs > vmax) vn = vn * vmax / vabs;
  return vn;
}

// ---- Anderson mixing of the viscosity iteration (picard_anderson_m > 0) --------------
// No counterpart in the reference, whose update is the relaxation :1499-1529.  The map is
// one unrelaxed Picard step, g(u) = velocity-limited solution of A(u) x = b(u); with the
// residual f = g(u) - u and the differences dF_i = f_i+1 - f_i, dG_i = g_i+1 - g_i of the
// last m iterations, the next iterate is g - sum_i gamma_i dG_i, gamma the least-squares
// minimiser of |f - sum_i gamma_i dF_i| (u on the cx points and v on the cy points make
// one vector).  k_aa_prepare writes g, f and the newest difference columns and reduces
// the inner products of the newest dF and of f with every history column; its last block
// updates the Gram matrix and solves for gamma on one thread; k_picard_update mixes.
struct AAArgs {
  Dims d;
  int m;
  double vmax;
  const double *u, *v, *xu, *xv;
  double *dFu[kAAMax], *dFv[kAAMax], *dGu[kAAMax], *dGv[kAAMax];
  double *fu, *fv, *gu, *gv;   // previous f, g on entry; this iteration's on exit
  double* sc;
  Reduction red;               // kAAPartials sums: dF_i . dF_new, then dF_i . f
};

__global__ void __launch_bounds__(256) k_aa_prepare(AAArgs a) {
  const Dims d = a.d;
  const bool have = a.sc[SC_AA_HAVE] != 0.0;
  const int s = (int)a.sc[SC_AA_HEAD];
  double acc[kAAPartials];
#pragma unroll
  for (int k = 0; k < kAAPartials; ++k) acc[k] = 0.0;
  FOR_TILES(d) {
    const long long q = d.at(j, i);
    auto point = [&](double g, double x, double* fp, double* gp, double* const* dF, double* const* dG) {
      const double f = g - x;
      if (have) {
        const double df = f - fp[q];
#pragma unroll
        for (int k = 0; k < kAAMax; ++k)
          if (k == s) {
            dF[k][q] = df;
            dG[k][q] = g - gp[q];
          }
#pragma unroll
        for (int k = 0; k < kAAMax; ++k) {
          if (k < a.m) {
            const double c = (k == s) ? df : dF[k][q];
            acc[k] += c * df;
            acc[kAAMax + k] += c * f;
          }
        }
      }
      fp[q] = f;
      gp[q] = g;
    };
    if (i < d.nx - 1) point(limited_u(d, a.xu, a.xv, a.vmax, j, i), a.u[q], a.fu, a.gu, a.dFu, a.dGu);
    if (j < d.ny - 1) point(limited_v(d, a.xu, a.xv, a.vmax, j, i), a.v[q], a.fv, a.gv, a.dFv, a.dGv);
  }
  // one thread: the Gram matrix update and the mixing coefficients (shared with the oracle's
  // restatement)
  if (reduce_all(acc, a.red)) aa_coefficients(a.sc, a.m, acc);
}

struct UpdArgs {
  Dims d;
  int diva, sliding_none, basal_freezing;
  double vmax, rel, dT_freeze;
  const double *xu, *xv;           // linear solution
  double *u, *v, *up, *vp;         // velocities (relaxed in place) and the previous iterate
  // Anderson mixing (aa_m > 0): the iterate is g - sum gamma_i dG_i instead of the relaxation
  int aa_m;
  double* sc;
  const double *gu, *gv;
  const double *dGu[kAAMax], *dGv[kAAMax];
  const double *uchk, *vchk;       // fields tested by estimate_visc_iter_UV_errors
  double *errx, *erry;             // DIVA_err candidates
  double *fex, *fey;               // DIVA_err: the previous iteration's candidate, if `commit`
  int commit;
  const double *bex, *bey, *F2, *Hi, *Ti, *Tpmp;
  double *taubx, *tauby, *ubx, *vby;
  Reduction red;                   // 3 sums
  IterEnd end;
};

// The loop's totals and whether it goes on (thread 0 of one block).
__device__ __forceinline__ void loop_end(double* sc, const IterEnd& e) {
  sc[SC_SUM_LIN] += sc[SC_LIN_IT];
  sc[SC_SUM_FULL] += sc[SC_LIN_FULL];
  sc[SC_N_SOLVED] += sc[SC_SOLVED];
  const bool stop = sc[SC_CONVERGED] != 0.0 || sc[SC_EXIT_RELRES] != 0.0 || sc[SC_NAN] != 0.0 ||
                    sc[SC_TIMEOUT] != 0.0 || sc[SC_PIC_IT] > (double)e.nit;
  cudaGraphSetConditional(e.a, stop ? 0u : 1u);
  if (e.has_b) cudaGraphSetConditional(e.b, stop ? 0u : 1u);
}

__global__ void __launch_bounds__(256) k_picard_update(UpdArgs a) {
  const Dims d = a.d;
  double sums[3] = {0.0, 0.0, 0.0};
  const bool commit = a.commit < 0 ? a.sc[SC_PIC_IT] > 1.0 : a.commit != 0;
  FOR_TILES(d) {
    const long long q = d.at(j, i);
    const bool cx = i < d.nx - 1, cy = j < d.ny - 1, aa = a.aa_m > 0, off = aa && a.sc[SC_AA_OFF] != 0.0;
    // every load of the point's two faces, then their stores
    bool frozen = false;
    if (a.diva && a.basal_freezing) {
      const long long ob = (long long)(d.nz - 1) * d.plane + q;
      frozen = a.Tpmp[ob] - a.Ti[ob] > a.dT_freeze;
    }
    const bool base = a.diva && !a.sliding_none;
    const double F20 = base ? a.F2[q] : 0.0, H0 = base ? a.Hi[q] : 0.0;
    struct Face { double old, now, last, chk, be, F2; } f[2] = {};
    auto read = [&](Face& f, const double* x, const double* g, const double* const* dG, const double* chk,
                    const double* err, const double* be, long long q1, auto limited) {
      f.old = x[q];
      if (aa) f.now = g[q];
      else f.now = limited();
      if (aa && !off)
        for (int k = 0; k < a.aa_m; ++k) f.now -= a.sc[SC_AA_GAMMA + k] * dG[k][q];
      else
        f.now = a.rel * f.now + (1.0 - a.rel) * f.old;   // (mixing given up: the relaxation of g)
      f.last = commit ? err[q] : 0.0;
      f.chk = a.diva ? f.now : chk[q];
      f.be = a.diva ? be[q] : 0.0;
      f.F2 = base ? stag_margin(F20, a.F2[q1], H0, a.Hi[q1]) : 0.0;
    };
    if (cx)
      read(f[0], a.u, a.gu, a.dGu, a.uchk, a.errx, a.bex, d.at(j, i + 1),
           [&] { return limited_u(d, a.xu, a.xv, a.vmax, j, i); });
    if (cy)
      read(f[1], a.v, a.gv, a.dGv, a.vchk, a.erry, a.bey, d.at(j + 1, i),
           [&] { return limited_v(d, a.xu, a.xv, a.vmax, j, i); });
    auto write = [&](const Face& f, double* x, double* prev, double* err, double* fe, double* taub, double* ub) {
      prev[q] = f.old;
      x[q] = f.now;
      if (fabs(f.now) > kVelTol) {
        sums[2] += 1.0;
        sums[0] += (f.now - f.old) * (f.now - f.old);
        sums[1] += (f.now + f.old) * (f.now + f.old);
      }
      if (commit) fe[q] = f.last;
      err[q] = (fabs(f.chk) > kVelTol) ? 2.0 * fabs(f.now - f.old) / fabs(f.now + f.old + 1E-5) : 0.0;
      if (a.diva) {
        const double tb = f.be * f.now;
        taub[q] = tb;
        ub[q] = a.sliding_none || frozen ? 0.0 : f.now - tb * f.F2;
      }
    };
    if (cx) write(f[0], a.u, a.up, a.errx, a.fex, a.taubx, a.ubx);
    if (cy) write(f[1], a.v, a.vp, a.erry, a.fey, a.tauby, a.vby);
  }
  if (!reduce_all(sums, a.red)) return;
  double* sc = a.sc;
  sc[SC_RES1] = sums[0];
  sc[SC_RES2] = sums[1];
  sc[SC_RES1 + 2] = sums[2];
  if (!a.end.graph) return;
  // the step norm (calc_visc_iter_UV_resid :1588-1596) and the stop test (:346-351)
  if (sc[SC_RNORM2] > sc[SC_TARGET2]) sc[SC_LIN_FAILED] += 1.0;
  if (!isfinite(sums[0]) || !isfinite(sums[1])) sc[SC_NAN] = 1.0;
  const double resid = (sums[2] > 0.0) ? 2.0 * sqrt(sums[0]) / max_ref(sqrt(sums[1]), 1E-8) : 0.0;
  sc[SC_RESID] = resid;
  sc[SC_CONVERGED] = ((a.end.loop && resid < a.end.tol) || sc[SC_PIC_IT] >= (double)a.end.nit) ? 1.0 : 0.0;
  if (a.end.loop) loop_end(sc, a.end);
}

// basal stress and velocity of the faces of point (j,i)
__device__ __forceinline__ void basal_point(const Dims& d, int sliding_none, int basal_freezing, double dT,
                                            const double* u, const double* v, const double* bex, const double* bey,
                                            const double* F2, const double* Hi, const double* Ti, const double* Tpmp,
                                            double* tbx, double* tby, double* ubx, double* vby, int j, int i) {
  const long long q = d.at(j, i);
  bool frozen = false;
  if (basal_freezing) {
    const long long ob = (long long)(d.nz - 1) * d.plane + q;
    frozen = Tpmp[ob] - Ti[ob] > dT;
  }
  if (i < d.nx - 1) {
    const double tb = bex[q] * u[q];
    tbx[q] = tb;
    const double F2s = stag_margin(F2[q], F2[d.at(j, i + 1)], Hi[q], Hi[d.at(j, i + 1)]);
    ubx[q] = sliding_none ? 0.0 : (frozen ? 0.0 : u[q] - tb * F2s);
  }
  if (j < d.ny - 1) {
    const double tb = bey[q] * v[q];
    tby[q] = tb;
    const double F2s = stag_margin(F2[q], F2[d.at(j + 1, i)], Hi[q], Hi[d.at(j + 1, i)]);
    vby[q] = sliding_none ? 0.0 : (frozen ? 0.0 : v[q] - tb * F2s);
  }
}

// calc_basal_stress + calc_basal_velocities at the current velocities (used when
// the viscosity iteration stops on the nonlinear residual before a linear solve)
__global__ void k_basal_stress_velocities(Dims d, int sliding_none, int basal_freezing, double dT, const double* u,
                                          const double* v, const double* bex, const double* bey, const double* F2,
                                          const double* Hi, const double* Ti, const double* Tpmp, double* tbx,
                                          double* tby, double* ubx, double* vby) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
  if (j >= d.ny || i >= d.nx) return;
  basal_point(d, sliding_none, basal_freezing, dT, u, v, bex, bey, F2, Hi, Ti, Tpmp, tbx, tby, ubx, vby, j, i);
}
// The post kernel of a graph-launched iteration under the rel-res stop rule: when the nonlinear
// residual ended it before a linear solve, the last DIVA_err candidate becomes the field and
// [DIVA] the basal stress and velocities are formed at the current velocities; the loop's
// handles are set either way.
__global__ void k_relres_end(Dims d, int diva, int sliding_none, int basal_freezing, double dT, const double* u,
                             const double* v, const double* bex, const double* bey, const double* F2,
                             const double* Hi, const double* Ti, const double* Tpmp, double* tbx, double* tby,
                             double* ubx, double* vby, const double* cx, const double* cy, double* fx, double* fy,
                             double* sc, IterEnd end) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
  const bool stopped = sc[SC_EXIT_RELRES] != 0.0;
  if (j == 0 && i == 0) loop_end(sc, end);   // (writes nothing that the other threads read)
  if (j >= d.ny || i >= d.nx || !stopped) return;
  const long long q = d.at(j, i);
  if (sc[SC_PIC_IT] > 1.0) {
    fx[q] = cx[q];
    fy[q] = cy[q];
  }
  if (diva) basal_point(d, sliding_none, basal_freezing, dT, u, v, bex, bey, F2, Hi, Ti, Tpmp, tbx, tby, ubx, vby, j, i);
}

// visc_eff_3D_b of the last viscosity iteration (:820-858), written once per solve
__global__ void k_visc_b(Dims d, int bc_margin, const double* visc, const int* mask_ice, double* vb) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y, k0 = blockIdx.z * kLayers;
  if (j >= d.ny - 1 || i >= d.nx - 1) return;
  const long long q = d.at(j, i), q1 = d.at(j, i + 1), q2 = d.at(j + 1, i), q3 = d.at(j + 1, i + 1);
  int m0 = 1, m1 = 1, m2 = 1, m3 = 1;
  double w = 0.0;
  if (bc_margin) {
    m0 = mask_ice[q] == 1; m1 = mask_ice[q1] == 1; m2 = mask_ice[q2] == 1; m3 = mask_ice[q3] == 1;
    w = (double)m0 + (double)m1 + (double)m2 + (double)m3;
  }
  double f0[kLayers], f1[kLayers], f2[kLayers], f3[kLayers];
  LOAD_LAYERS(e, k, k0, d.nz) {
    const double* f = visc + k * d.plane;
    f0[e] = f[q]; f1[e] = f[q1]; f2[e] = f[q2]; f3[e] = f[q3];
  }
  FOR_LAYERS(e, k0, d.nz) {
    double s;
    if (bc_margin) {
      s = 0.0;
      if (m0) s = s + f0[e];
      if (m1) s = s + f1[e];
      if (m2) s = s + f2[e];
      if (m3) s = s + f3[e];
      if (w > 0.0) s = s / w;
    } else {
      s = (f0[e] + f1[e] + f2[e] + f3[e]) / 4.0;
    }
    vb[(k0 + e) * d.plane + q] = s;
  }
}

// F1(zeta) = int_base^zeta (-H/eta) zeta dzeta on the a-grid (:1222-1227)
__global__ void k_f1(Dims d, Zeta zt, const double* Hi, const double* visc, double* F1) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
  if (j >= d.ny || i >= d.nx) return;
  const long long q = d.at(j, i);
  const double H = Hi[q];
  const int nz = d.nz;
  double acc = 0.0, fk1 = 0.0;
  for (int k0 = 0; k0 < nz; k0 += kLayers) {   // from the base up
    double f[kLayers];
    LOAD_LAYERS(e, k, k0, nz) f[e] = visc[(nz - 1 - k) * d.plane + q];
    FOR_LAYERS(e, k0, nz) {
      const int k = nz - 1 - k0 - e;
      const double fk = (-H / f[e]) * zt.z[k];
      if (k < nz - 1) acc = acc - 0.5 * (fk1 + fk) * (zt.z[k + 1] - zt.z[k]);
      F1[(long long)k * d.plane + q] = acc;
      fk1 = fk;
    }
  }
}

// u_3D = u_base + taub * F1_stag (:1229-1289)
__global__ void k_u3d(Dims d, int bc_margin, const double* Hi, const double* F1, const double* ubx, const double* vby,
                      const double* tbx, const double* tby, double* u3, double* v3) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y, k0 = blockIdx.z * kLayers;
  if (j >= d.ny || i >= d.nx) return;
  const long long q = d.at(j, i);
  const bool cx = i < d.nx - 1, cy = j < d.ny - 1;
  const double H0 = Hi[q], He = cx ? Hi[q + d.ld] : 0.0, Hn = cy ? Hi[q + 1] : 0.0;
  const double ub = cx ? ubx[q] : 0.0, tx = cx ? tbx[q] : 0.0, vb = cy ? vby[q] : 0.0, ty = cy ? tby[q] : 0.0;
  const long long qe = cx ? q + d.ld : q, qn = cy ? q + 1 : q;
  double f[kLayers], fe[kLayers], fn[kLayers];
  LOAD_LAYERS(e, k, k0, d.nz) {
    const double* F = F1 + k * d.plane;
    f[e] = F[q]; fe[e] = F[qe]; fn[e] = F[qn];
  }
  auto staggered = [&](double H1, double f0, double f1) {
    if (!bc_margin) return 0.5 * (f0 + f1);
    if (H0 > 0.0 && H1 == 0.0) return f0;
    if (H0 == 0.0 && H1 > 0.0) return f1;
    return H0 > 0.0 && H1 > 0.0 ? 0.5 * (f0 + f1) : 0.0;
  };
  FOR_LAYERS(e, k0, d.nz) {
    const long long o = (k0 + e) * d.plane + q;
    if (cx) u3[o] = ub + tx * staggered(He, f[e], fe[e]);
    if (cy) v3[o] = vb + ty * staggered(Hn, f[e], fn[e]);
  }
}

// Per-face part of calc_secondary_velocities (:393-485): the 3D cx/cy fields per
// mode, base velocities, surface velocities and (SIA, SIA/SSA) vertical averages.
__global__ void k_faces_prelude(Dims d, Zeta zt, int dyn, double* u3, double* v3, const double* u3s,
                                const double* v3s, const double* uS, const double* vS, double* ub, double* vb,
                                double* us, double* vs, double* uv, double* vv) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
  if (j >= d.ny || i >= d.nx) return;
  const long long q = d.at(j, i);
  for (int face = 0; face < 2; ++face) {
    if (face == 0 && i >= d.nx - 1) continue;
    if (face == 1 && j >= d.ny - 1) continue;
    double* f3 = face == 0 ? u3 : v3;
    const double* s3 = face == 0 ? u3s : v3s;
    const double sS = face == 0 ? uS[q] : vS[q];
    double* base = face == 0 ? ub : vb;
    double* surf = face == 0 ? us : vs;
    double* vav = face == 0 ? uv : vv;
    // the layers this face has: its own, or made here
    const bool own = dyn != DIVA_DYN_SIA && dyn != DIVA_DYN_SSA && dyn != DIVA_DYN_SIA_SSA;
    const bool mean = dyn == DIVA_DYN_SIA || dyn == DIVA_DYN_SIA_SSA;
    if (own) {
      surf[q] = f3[q];
      continue;
    }
    base[q] = dyn == DIVA_DYN_SIA ? 0.0 : sS;
    if (dyn == DIVA_DYN_SSA) vav[q] = sS;
    double avg = 0.0, prev = 0.0;
    for (int k0 = 0; k0 < d.nz; k0 += kLayers) {
      double f[kLayers];
      LOAD_LAYERS(e, k, k0, d.nz) f[e] = dyn == DIVA_DYN_SSA ? sS : s3[k * d.plane + q];
      FOR_LAYERS(e, k0, d.nz) {
        const int k = k0 + e;
        if (dyn == DIVA_DYN_SIA_SSA) f[e] = f[e] + sS;
        f3[k * d.plane + q] = f[e];
        if (k == 0) surf[q] = f[e];
        else avg = avg + 0.5 * (f[e] + prev) * (zt.z[k] - zt.z[k - 1]);
        prev = f[e];
      }
    }
    if (mean) vav[q] = avg;
  }
}

struct SecArgs {
  Dims d;
  Zeta zt;
  int dyn;
  const double *u3, *v3, *Hs, *Hi, *dHs_dx, *dHs_dy, *dHi_dx, *dHi_dy, *dHb_dt;
  const double *uv, *vv, *us, *vs, *ub, *vb;
  const int *sheet, *ice;
  double *w, *ws, *wb, *u3a, *v3a, *uva, *vva, *usa, *vsa, *uba, *vba, *abv, *abs_, *abb, *Rs;
};

// map_velocity_from_cx_to_a, ..cy_to_a (:2592-2811) at a point: which of the two neighbouring
// faces its value comes from, by the ice mask along the direction: 0 none, 1 the first (west or
// south), 2 the second, 3 their mean.  At the grid's ends the one face there is: the first of
// the pair (0, 1) at the start, the second of the last pair at the end.
__device__ __forceinline__ int map_mode(const int* ice, long long q, long long step, bool start, bool end) {
  const bool m1 = ice[q] == 1;
  const int m0 = ice[start ? q : q - step], m2 = ice[end ? q : q + step];
  if (!m1) return 0;
  if (start) return 1;
  if (end) return 2;
  if (m0 == 1) return m2 == 1 ? 3 : (m2 == 0 ? 1 : 0);
  return m0 == 0 && m2 == 1 ? 2 : 0;
}
__device__ __forceinline__ double map_faces(int mode, double f0, double f1) {
  return mode == 3 ? 0.5 * (f0 + f1) : mode == 2 ? f1 : mode == 1 ? f0 : 0.0;
}

// W: the vertical velocities too (not in SSA).  Bound by memory: with them five 3D fields are read
// and three written.
template <bool W>
__global__ void __launch_bounds__(256, 2) k_secondary(SecArgs a) {
  const Dims d = a.d;
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
  if (j >= d.ny || i >= d.nx) return;
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  const long long q = d.at(j, i), P = d.plane;
  const double dx = d.dx;
  double dHbase_dx = 0.0, dHbase_dy = 0.0;
  if (W) {
    // calc_3D_vertical_velocities :562-650; surface/thickness slopes recomputed from Hs, Hi (:563-566)
    auto A = [&](const double* f, int jj, int ii) { return f[d.at(jj, ii)]; };
    double sx, sy, hx, hy;
    if (i > 0 && i < nx - 1) { sx = (A(a.Hs, j, i + 1) - A(a.Hs, j, i - 1)) / (2 * dx); hx = (A(a.Hi, j, i + 1) - A(a.Hi, j, i - 1)) / (2 * dx); }
    else if (i == 0) { sx = (A(a.Hs, j, 1) - A(a.Hs, j, 0)) / dx; hx = (A(a.Hi, j, 1) - A(a.Hi, j, 0)) / dx; }
    else { sx = (A(a.Hs, j, nx - 1) - A(a.Hs, j, nx - 2)) / dx; hx = (A(a.Hi, j, nx - 1) - A(a.Hi, j, nx - 2)) / dx; }
    if (j > 0 && j < ny - 1) { sy = (A(a.Hs, j + 1, i) - A(a.Hs, j - 1, i)) / (2 * dx); hy = (A(a.Hi, j + 1, i) - A(a.Hi, j - 1, i)) / (2 * dx); }
    else if (j == 0) { sy = (A(a.Hs, 1, i) - A(a.Hs, 0, i)) / dx; hy = (A(a.Hi, 1, i) - A(a.Hi, 0, i)) / dx; }
    else { sy = (A(a.Hs, ny - 1, i) - A(a.Hs, ny - 2, i)) / dx; hy = (A(a.Hi, ny - 1, i) - A(a.Hi, ny - 2, i)) / dx; }
    dHbase_dx = sx - hx;
    dHbase_dy = sy - hy;
  }
  // the faces of the divergence stencil in x and y (:603-622), which the a-grid maps read as well
  const int ia = (i == 0) ? 1 : (i == nx - 1 ? nx - 2 : i), ja = (j == 0) ? 1 : (j == ny - 1 ? ny - 2 : j);
  const long long qe = d.at(j, ia), qw = d.at(j, ia - 1), qn = d.at(ja, i), qs = d.at(ja - 1, i);
  const int mx = map_mode(a.ice, q, d.ld, i == 0, i == nx - 1), my = map_mode(a.ice, q, 1, j == 0, j == ny - 1);
  double Hdx = 0.0, Hr = 0.0, gsx = 0.0, gsy = 0.0, gix = 0.0, giy = 0.0;
  if (W) {
    const double H = a.Hi[q];
    Hdx = H / (2.0 * dx); Hr = H / max_ref(0.1, H);
    gsx = a.dHs_dx[q]; gsy = a.dHs_dy[q]; gix = a.dHi_dx[q]; giy = a.dHi_dy[q];
  }
  // From the base up; a layer's a-grid velocities are read (stale) for w before they are replaced.
  // w_k = w_k+1 - H ((du/dx + dv/dy) + (dHs/dx - zm dHi/dx) / H du/dz + ..) dz with the means of
  // both layers, dx, H and dz taken out of the sums: no division in a layer (six cost 500
  // instructions a layer, 3/4 of the kernel).
  double wk1 = 0.0, div_kp1 = 0.0, ua_kp1 = 0.0, va_kp1 = 0.0;
  for (int k0 = 0; k0 < nz; k0 += kLayers) {
    double ue[kLayers], uw[kLayers], vn[kLayers], vs[kLayers], ua[kLayers], va[kLayers];
    LOAD_LAYERS(e, kb, k0, nz) {
      const long long o = (nz - 1 - kb) * P;
      ue[e] = a.u3[o + qe]; uw[e] = a.u3[o + qw]; vn[e] = a.v3[o + qn]; vs[e] = a.v3[o + qs];
      if (W) { ua[e] = a.u3a[o + q]; va[e] = a.v3a[o + q]; }
    }
    FOR_LAYERS(e, k0, nz) {
      const int k = nz - 1 - k0 - e;
      const long long o = k * P;
      if (W) {
        const double div = (ue[e] - uw[e]) + (vn[e] - vs[e]);
        if (k == nz - 1) {
          const double ubase = i == 0 ? uw[e] : i == nx - 1 ? ue[e] : 0.5 * (uw[e] + ue[e]);
          const double vbase = j == 0 ? vs[e] : j == ny - 1 ? vn[e] : 0.5 * (vs[e] + vn[e]);
          wk1 = (ubase * dHbase_dx) + (vbase * dHbase_dy);
          if (a.sheet[q] == 1) wk1 = wk1 + a.dHb_dt[q];
          a.wb[q] = wk1;
        } else {
          const double dz = a.zt.z[k + 1] - a.zt.z[k], zm = 0.5 * (a.zt.z[k + 1] + a.zt.z[k]);
          const double tilt = (gsx - zm * gix) * (ua_kp1 - ua[e]) + (gsy - zm * giy) * (va_kp1 - va[e]);
          wk1 = wk1 - (Hdx * dz * (div + div_kp1) + Hr * tilt);
        }
        a.w[o + q] = wk1;
        if (k == 0) a.ws[q] = wk1;
        div_kp1 = div; ua_kp1 = ua[e]; va_kp1 = va[e];
      }
      a.u3a[o + q] = map_faces(mx, uw[e], ue[e]);
      a.v3a[o + q] = map_faces(my, vs[e], vn[e]);
    }
  }
  auto map_x = [&](const double* f) { return map_faces(mx, f[qw], f[qe]); };
  auto map_y = [&](const double* f) { return map_faces(my, f[qs], f[qn]); };
  const double uva = map_x(a.uv), vva = map_y(a.vv), usa = map_x(a.us), vsa = map_y(a.vs);
  const double uba = map_x(a.ub), vba = map_y(a.vb);
  a.uva[q] = uva; a.vva[q] = vva; a.usa[q] = usa; a.vsa[q] = vsa; a.uba[q] = uba; a.vba[q] = vba;
  const double av = sqrt(uva * uva + vva * vva), as = sqrt(usa * usa + vsa * vsa), ab = sqrt(uba * uba + vba * vba);
  a.abv[q] = av; a.abs_[q] = as; a.abb[q] = ab;
  double R;
  if (a.dyn == DIVA_DYN_SIA) R = 1.0;
  else if (a.dyn == DIVA_DYN_SSA) R = 0.0;
  else R = (a.ice[q] == 1) ? max_ref(0.0, min_ref(1.0, (1.0 - ab / as))) : 0.0;
  a.Rs[q] = R;
}

// solve_SIA 3D velocities (:60-105)
__global__ void k_sia(Dims d, Zeta zt, double n, const int* sheet, const double* Hcx, const double* Hcy,
                      const double* sxcx, const double* sycx, const double* sxcy, const double* sycy,
                      const double* Acx, const double* Acy, double* u3, double* v3) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
  if (j >= d.ny || i >= d.nx) return;
  const long long q = d.at(j, i), P = d.plane;
  const int nz = d.nz;
  for (int face = 0; face < 2; ++face) {
    if (face == 0 && i >= d.nx - 1) continue;
    if (face == 1 && j >= d.ny - 1) continue;
    const long long qn = face == 0 ? d.at(j, i + 1) : d.at(j + 1, i);
    double* out = face == 0 ? u3 : v3;
    if (sheet[q] == 0 && sheet[qn] == 0) {
      for (int k = 0; k < nz; ++k) out[(long long)k * P + q] = 0.0;
      continue;
    }
    const double H = face == 0 ? Hcx[q] : Hcy[q];
    const double sx = face == 0 ? sxcx[q] : sxcy[q], sy = face == 0 ? sycx[q] : sycy[q];
    const double* A = face == 0 ? Acx : Acy;
    const double slope = face == 0 ? sx : sy;
    const double D0 = pow(kRhoI * kGrav * H, n) * pow((sx * sx + sy * sy), (n - 1.0) / 2.0);
    // D(zeta) = 2 H int_base^zeta A zeta^n (vertical_integration_from_bottom_to_zeta)
    double acc = 0.0, fk1 = 0.0;
    for (int k0 = 0; k0 < nz; k0 += kLayers) {   // from the base up
      double f[kLayers];
      LOAD_LAYERS(e, k, k0, nz) f[e] = A[(nz - 1 - k) * P + q];
      FOR_LAYERS(e, k0, nz) {
        const int k = nz - 1 - k0 - e;
        const double fk = f[e] * zt.zn[k];
        if (k < nz - 1) acc = acc - 0.5 * (fk1 + fk) * (zt.z[k + 1] - zt.z[k]);
        out[k * P + q] = max_ref(D0 * (2.0 * H * acc), -1E5) * slope;
        fk1 = fk;
      }
    }
  }
}

__global__ void k_count_sheet(Dims d, const int* sheet, int* out) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
  if (j >= d.ny || i >= d.nx) return;
  if (sheet[d.at(j, i)] != 0) atomicOr(out, 1);
}

__global__ void k_zero_uv(Dims d, double* u, double* v) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
  if (j >= d.ny || i >= d.nx) return;
  if (i < d.nx - 1) u[d.at(j, i)] = 0.0;
  if (j < d.ny - 1) v[d.at(j, i)] = 0.0;
}

}  // namespace

#define G2 grid2d(c->d.ny, c->d.nx), block2d(), 0, c->stream
#define G3 grid_layers(c->d.ny, c->d.nx, c->d.nz), block2d(), 0, c->stream

// Whether K1 computes the viscosity of the linearisation in FP32 (precision 'mixed').
#ifndef DIVA_K1_FP32
#define DIVA_K1_FP32 1
#endif
static bool k1_fp32(const diva_config_t& C) { return DIVA_K1_FP32 && C.precision == DIVA_PREC_MIXED; }

int launch_prepare_afac(Ctx* c) {
  k_afac<<<G3>>>(c->d, c->c.n_flow, c->D(DIVA_F_A_FLOW_3D_A), c->afac); c->launches++;
  DIVA_LAUNCHED(c, "k_afac");
  return DIVA_OK;
}

static void fill_coef_args(Ctx* c, CoefArgs& a, const double* u, const double* v, bool diva) {
  const diva_config_t& C = c->c;
  a.d = c->d;
  a.zt = c->zt;
  a.diva = diva;
  a.bc_margin = C.choice_ice_margin == DIVA_MARGIN_BC;
  a.sliding = C.choice_sliding_law;
  a.gl_subgrid = C.do_GL_subgrid_friction;
  a.basal_freezing = C.include_basal_freezing;
  a.prescribed_tauc = C.prescribed_tauc;
  a.n_is_3 = C.n_flow == 3.0;
  a.crossterms = C.include_SSADIVA_crossterms;
  a.n_flow = C.n_flow;
  a.eps0 = C.DIVA_epsilon_sq_0;
  a.visc_min = C.DIVA_visc_eff_min;
  a.beta_max = C.DIVA_beta_max;
  a.delta_v = C.slid_delta_v;
  a.wm = C.slid_Weertman_m;
  a.q_plastic = C.slid_Coulomb_reg_q_plastic;
  a.u_thr = C.slid_Coulomb_reg_u_threshold;
  a.zi_ut = C.slid_ZI_ut;
  a.zi_p = C.slid_ZI_p;
  a.dT_freeze = C.deltaT_basal_freezing;
  {
    // F_int_min = vertical_integrate( (1/visc_eff_min) * zeta**2) (:980)
    double s = 0.0;
    for (int k = 1; k < c->d.nz; ++k) {
      const double f0 = (1.0 / C.DIVA_visc_eff_min) * c->zt.z2[k - 1], f1 = (1.0 / C.DIVA_visc_eff_min) * c->zt.z2[k];
      s = s + 0.5 * (f1 + f0) * (c->zt.z[k] - c->zt.z[k - 1]);
    }
    a.Fmin = s;
  }
  a.u = u; a.v = v;
  a.visc_prev = c->visc_prev;
  a.taub_cx = c->D(DIVA_F_TAUB_CX); a.taub_cy = c->D(DIVA_F_TAUB_CY);
  a.Hi = c->D(DIVA_F_HI_A); a.afac = c->afac;
  a.mask_ice = c->I(DIVA_F_MASK_ICE_A); a.mask_ocean = c->I(DIVA_F_MASK_OCEAN_A);
  a.beta_sq = c->D(DIVA_F_BETA_SQ_A); a.phi_fric = c->D(DIVA_F_PHI_FRIC_A); a.alpha_sq = c->D(DIVA_F_ALPHA_SQ_A);
  a.Neff = c->D(DIVA_F_NEFF_A); a.Ti = c->D(DIVA_F_TI_A); a.Tpmp = c->D(DIVA_F_TI_PMP_A);
  a.dudz = c->D(DIVA_F_DU_DZ_3D_CX); a.dvdz = c->D(DIVA_F_DV_DZ_3D_CY);
  a.visc = c->D(DIVA_F_VISC_EFF_3D_A); a.visc_int = c->D(DIVA_F_VISC_EFF_INT_A); a.Na = c->D(DIVA_F_N_A);
  a.beta = c->D(DIVA_F_BETA_A); a.F2 = c->D(DIVA_F_F2_A); a.beta_eff = c->D(DIVA_F_BETA_EFF_A);
  a.tauc = c->D(DIVA_F_TAUC_A);
  a.col_eps = c->col_eps;
  a.col_flags = c->col_flags;
  a.taub_seen_cx = c->taub_seen[0];
  a.taub_seen_cy = c->taub_seen[1];
}

int launch_diva_coefficients(Ctx* c, const double* u, const double* v, bool diva, int what, bool begin) {
  const diva_config_t& C = c->c;
  // Picard double buffering of visc_eff_3D_a: read the previous, write the new
  std::swap(c->f[DIVA_F_VISC_EFF_3D_A], *reinterpret_cast<void**>(&c->visc_prev));
  CoefArgs a{};
  fill_coef_args(c, a, u, v, diva);
  if (C.choice_ice_margin == DIVA_MARGIN_BC) {
    // BC margins keep visc_eff_int_a / N_a of ice-free points from before: the
    // previous buffer's content is not carried over by the swap, so copy it.
    DIVA_CUDA(c, cudaMemcpyAsync(c->D(DIVA_F_VISC_EFF_3D_A), c->visc_prev, sizeof(double) * c->d.plane * c->d.nz,
                                 cudaMemcpyDeviceToDevice, c->stream));
  }
  a.keep_seen = what != K1_WRITE_SHEAR;
  a.sc = begin ? c->scal : nullptr;
  k_column_prep<<<G2>>>(a); c->launches++;
  {
    const dim3 block(kColLanes, kColRows);
    const int L = visc_layers(c->d);
    const dim3 grid((c->d.nz + L - 1) / L, (c->d.ny + kColLanes - 1) / kColLanes, (c->d.nx + kColRows - 1) / kColRows);
    const bool f32 = k1_fp32(C), w = what == K1_WRITE_SHEAR;
    auto kern = w ? (f32 ? (L == 1 ? k_layer_viscosity<true, float, 1> : k_layer_viscosity<true, float, kViscLayers>)
                         : (L == 1 ? k_layer_viscosity<true, double, 1> : k_layer_viscosity<true, double, kViscLayers>))
                  : (f32 ? (L == 1 ? k_layer_viscosity<false, float, 1> : k_layer_viscosity<false, float, kViscLayers>)
                         : (L == 1 ? k_layer_viscosity<false, double, 1> : k_layer_viscosity<false, double, kViscLayers>));
    kern<<<grid, block, 0, c->stream>>>(a);
    c->launches++;
  }
  if (k1_fp32(C)) {
    if (c->d.nz == 15) k_column_integrals<15, float><<<G2>>>(a);
    else k_column_integrals<0, float><<<G2>>>(a);
  } else {
    if (c->d.nz == 15) k_column_integrals<15, double><<<G2>>>(a);
    else k_column_integrals<0, double><<<G2>>>(a);
  }
  c->launches++;
  if (what == K1_COLUMNS_ONLY) {   // timing of the column launches alone (diva_profile_kernel)
    DIVA_LAUNCHED(c, "column coefficients");
    return DIVA_OK;
  }
  DIVA_LAUNCHED(c, "column coefficients");
  FaceArgs fa{};
  fa.d = c->d;
  fa.bc_margin = a.bc_margin;
  fa.apply_fgrnd = diva ? C.do_GL_subgrid_friction : 1;   // solve_SSA always applies f_grnd^2 (:200-205)
  fa.crossterms = C.include_SSADIVA_crossterms;
  fa.vint = c->D(DIVA_F_VISC_EFF_INT_A); fa.Hb_i = c->D(DIVA_F_HI_B); fa.beta_eff = c->D(DIVA_F_BETA_EFF_A);
  fa.fcx = c->D(DIVA_F_F_GRND_CX); fa.fcy = c->D(DIVA_F_F_GRND_CY); fa.Na = c->D(DIVA_F_N_A);
  fa.mask_ice = c->I(DIVA_F_MASK_ICE_A);
  fa.visc_int_b = c->D(DIVA_F_VISC_EFF_INT_B); fa.Nb = c->D(DIVA_F_N_B);
  fa.bex = c->D(DIVA_F_BETA_EFF_CX); fa.bey = c->D(DIVA_F_BETA_EFF_CY);
  fa.Ncx = c->D(DIVA_F_N_CX); fa.Ncy = c->D(DIVA_F_N_CY);
  fa.lvBx = c->lv[0].Bx; fa.lvBy = c->lv[0].By; fa.lvNa = c->lv[0].Na; fa.lvNb = c->lv[0].Nb;
  k_face_coefficients<<<G2>>>(fa); c->launches++;
  DIVA_LAUNCHED(c, "k_face_coefficients");
  return DIVA_OK;
}

int launch_picard_update(Ctx* c, double* u, double* v, const double* xu, const double* xv, bool diva, int commit,
                         const IterEnd* end) {
  const diva_config_t& C = c->c;
  UpdArgs a{};
  a.d = c->d;
  a.diva = diva;
  a.sliding_none = C.choice_sliding_law == DIVA_SLIDING_NONE;
  a.basal_freezing = C.include_basal_freezing;
  a.vmax = C.DIVA_vel_max;
  a.rel = C.DIVA_visc_it_relax;
  a.dT_freeze = C.deltaT_basal_freezing;
  a.xu = xu; a.xv = xv; a.u = u; a.v = v;
  a.up = c->D(DIVA_F_U_CX_PREV); a.vp = c->D(DIVA_F_V_CY_PREV);
  a.uchk = c->D(DIVA_F_U_VAV_CX); a.vchk = c->D(DIVA_F_V_VAV_CY);
  a.errx = c->err_cand[0]; a.erry = c->err_cand[1];
  a.fex = c->D(DIVA_F_DIVA_ERR_CX); a.fey = c->D(DIVA_F_DIVA_ERR_CY);
  a.commit = commit;
  a.bex = c->D(DIVA_F_BETA_EFF_CX); a.bey = c->D(DIVA_F_BETA_EFF_CY); a.F2 = c->D(DIVA_F_F2_A);
  a.Hi = c->D(DIVA_F_HI_A); a.Ti = c->D(DIVA_F_TI_A); a.Tpmp = c->D(DIVA_F_TI_PMP_A);
  a.taubx = c->D(DIVA_F_TAUB_CX); a.tauby = c->D(DIVA_F_TAUB_CY);
  a.ubx = c->D(DIVA_F_U_BASE_CX); a.vby = c->D(DIVA_F_V_BASE_CY);
  a.red = Reduction{c->partials, c->red_count};
  if (end) a.end = *end;
  a.aa_m = C.picard_anderson_m;
  a.sc = c->scal;
  a.gu = c->aa_g[0]; a.gv = c->aa_g[1];
  for (int k = 0; k < kAAMax; ++k) { a.dGu[k] = c->aa_dG[k][0]; a.dGv[k] = c->aa_dG[k][1]; }
  k_picard_update<<<red_blocks(c->d), block2d(), 0, c->stream>>>(a); c->launches++;
  DIVA_LAUNCHED(c, "k_picard_update");
  return DIVA_OK;
}

int launch_anderson_prepare(Ctx* c, const double* u, const double* v, const double* xu, const double* xv) {
  const diva_config_t& C = c->c;
  AAArgs a{};
  a.d = c->d;
  a.m = C.picard_anderson_m;
  a.vmax = C.DIVA_vel_max;
  a.u = u; a.v = v; a.xu = xu; a.xv = xv;
  for (int k = 0; k < kAAMax; ++k) {
    a.dFu[k] = c->aa_dF[k][0]; a.dFv[k] = c->aa_dF[k][1];
    a.dGu[k] = c->aa_dG[k][0]; a.dGv[k] = c->aa_dG[k][1];
  }
  a.fu = c->aa_f[0]; a.fv = c->aa_f[1]; a.gu = c->aa_g[0]; a.gv = c->aa_g[1];
  a.sc = c->scal;
  a.red = Reduction{c->partials, c->red_count};
  k_aa_prepare<<<red_blocks(c->d), block2d(), 0, c->stream>>>(a); c->launches++;
  DIVA_LAUNCHED(c, "k_aa_prepare");
  return DIVA_OK;
}

// start of a solve: empty history, zeroed columns (unused slots then mix in nothing)
int anderson_reset(Ctx* c) {
  if (c->c.picard_anderson_m <= 0) return DIVA_OK;
  for (int q = 0; q < 2; ++q)
    for (int k = 0; k < kAAMax; ++k) {
      DIVA_CUDA(c, cudaMemsetAsync(c->aa_dF[k][q], 0, sizeof(double) * c->d.plane, c->stream));
      DIVA_CUDA(c, cudaMemsetAsync(c->aa_dG[k][q], 0, sizeof(double) * c->d.plane, c->stream));
    }
  return DIVA_OK;
}

int launch_commit_err(Ctx* c) {
  const size_t nb = sizeof(double) * c->d.plane;
  DIVA_CUDA(c, cudaMemcpyAsync(c->D(DIVA_F_DIVA_ERR_CX), c->err_cand[0], nb, cudaMemcpyDeviceToDevice, c->stream));
  DIVA_CUDA(c, cudaMemcpyAsync(c->D(DIVA_F_DIVA_ERR_CY), c->err_cand[1], nb, cudaMemcpyDeviceToDevice, c->stream));
  return DIVA_OK;
}

int launch_basal_stress_velocities(Ctx* c) {
  const diva_config_t& C = c->c;
  k_basal_stress_velocities<<<G2>>>(c->d, C.choice_sliding_law == DIVA_SLIDING_NONE, C.include_basal_freezing,
                                    C.deltaT_basal_freezing, c->D(DIVA_F_U_VAV_CX), c->D(DIVA_F_V_VAV_CY),
                                    c->D(DIVA_F_BETA_EFF_CX), c->D(DIVA_F_BETA_EFF_CY), c->D(DIVA_F_F2_A),
                                    c->D(DIVA_F_HI_A), c->D(DIVA_F_TI_A), c->D(DIVA_F_TI_PMP_A),
                                    c->D(DIVA_F_TAUB_CX), c->D(DIVA_F_TAUB_CY), c->D(DIVA_F_U_BASE_CX),
                                    c->D(DIVA_F_V_BASE_CY)); c->launches++;
  DIVA_LAUNCHED(c, "k_basal_stress_velocities");
  return DIVA_OK;
}

int launch_relres_end(Ctx* c, bool diva, const IterEnd& end) {
  const diva_config_t& C = c->c;
  k_relres_end<<<G2>>>(c->d, diva, C.choice_sliding_law == DIVA_SLIDING_NONE, C.include_basal_freezing,
                       C.deltaT_basal_freezing, c->D(DIVA_F_U_VAV_CX), c->D(DIVA_F_V_VAV_CY),
                       c->D(DIVA_F_BETA_EFF_CX), c->D(DIVA_F_BETA_EFF_CY), c->D(DIVA_F_F2_A), c->D(DIVA_F_HI_A),
                       c->D(DIVA_F_TI_A), c->D(DIVA_F_TI_PMP_A), c->D(DIVA_F_TAUB_CX), c->D(DIVA_F_TAUB_CY),
                       c->D(DIVA_F_U_BASE_CX), c->D(DIVA_F_V_BASE_CY), c->err_cand[0], c->err_cand[1],
                       c->D(DIVA_F_DIVA_ERR_CX), c->D(DIVA_F_DIVA_ERR_CY), c->scal, end); c->launches++;
  DIVA_LAUNCHED(c, "k_relres_end");
  return DIVA_OK;
}

int launch_shear_rates(Ctx* c) {
  CoefArgs a{};
  fill_coef_args(c, a, c->D(DIVA_F_U_VAV_CX), c->D(DIVA_F_V_VAV_CY), true);
  const dim3 block(kColLanes, kColRows);
  const dim3 grid(c->d.nz, (c->d.ny + kColLanes - 1) / kColLanes, (c->d.nx + kColRows - 1) / kColRows);
  if (k1_fp32(c->c)) k_shear_rates<float><<<grid, block, 0, c->stream>>>(a);
  else k_shear_rates<double><<<grid, block, 0, c->stream>>>(a);
  c->launches++;
  DIVA_LAUNCHED(c, "k_shear_rates");
  return DIVA_OK;
}

int launch_visc_b_output(Ctx* c) {
  // the shear strain rates the last viscosity iteration's K1 saw (the loop does not write them)
  int st;
  if ((st = launch_shear_rates(c))) return st;
  k_visc_b<<<G3>>>(c->d, c->c.choice_ice_margin == DIVA_MARGIN_BC, c->D(DIVA_F_VISC_EFF_3D_A),
                   c->I(DIVA_F_MASK_ICE_A), c->D(DIVA_F_VISC_EFF_3D_B)); c->launches++;
  DIVA_LAUNCHED(c, "k_visc_b");
  return DIVA_OK;
}

int launch_3d_horizontal_velocities(Ctx* c) {
  k_f1<<<G2>>>(c->d, c->zt, c->D(DIVA_F_HI_A), c->D(DIVA_F_VISC_EFF_3D_A), c->D(DIVA_F_F1_3D_A)); c->launches++;
  DIVA_LAUNCHED(c, "k_f1");
  k_u3d<<<G3>>>(c->d, c->c.choice_ice_margin == DIVA_MARGIN_BC, c->D(DIVA_F_HI_A), c->D(DIVA_F_F1_3D_A),
                c->D(DIVA_F_U_BASE_CX), c->D(DIVA_F_V_BASE_CY), c->D(DIVA_F_TAUB_CX), c->D(DIVA_F_TAUB_CY),
                c->D(DIVA_F_U_3D_CX), c->D(DIVA_F_V_3D_CY)); c->launches++;
  DIVA_LAUNCHED(c, "k_u3d");
  return DIVA_OK;
}

int launch_secondary_velocities(Ctx* c) {
  const int dyn = c->c.choice_ice_dynamics;
  k_faces_prelude<<<G2>>>(c->d, c->zt, dyn, c->D(DIVA_F_U_3D_CX), c->D(DIVA_F_V_3D_CY), c->D(DIVA_F_U_3D_SIA_CX),
                          c->D(DIVA_F_V_3D_SIA_CY), c->D(DIVA_F_U_SSA_CX), c->D(DIVA_F_V_SSA_CY),
                          c->D(DIVA_F_U_BASE_CX), c->D(DIVA_F_V_BASE_CY), c->D(DIVA_F_U_SURF_CX),
                          c->D(DIVA_F_V_SURF_CY), c->D(DIVA_F_U_VAV_CX), c->D(DIVA_F_V_VAV_CY)); c->launches++;
  DIVA_LAUNCHED(c, "k_faces_prelude");
  SecArgs a{};
  a.d = c->d; a.zt = c->zt; a.dyn = dyn;
  a.u3 = c->D(DIVA_F_U_3D_CX); a.v3 = c->D(DIVA_F_V_3D_CY); a.Hs = c->D(DIVA_F_HS_A); a.Hi = c->D(DIVA_F_HI_A);
  a.dHs_dx = c->D(DIVA_F_DHS_DX_A); a.dHs_dy = c->D(DIVA_F_DHS_DY_A);
  a.dHi_dx = c->D(DIVA_F_DHI_DX_A); a.dHi_dy = c->D(DIVA_F_DHI_DY_A); a.dHb_dt = c->D(DIVA_F_DHB_DT_A);
  a.uv = c->D(DIVA_F_U_VAV_CX); a.vv = c->D(DIVA_F_V_VAV_CY); a.us = c->D(DIVA_F_U_SURF_CX);
  a.vs = c->D(DIVA_F_V_SURF_CY); a.ub = c->D(DIVA_F_U_BASE_CX); a.vb = c->D(DIVA_F_V_BASE_CY);
  a.sheet = c->I(DIVA_F_MASK_SHEET_A); a.ice = c->I(DIVA_F_MASK_ICE_A);
  a.w = c->D(DIVA_F_W_3D_A); a.ws = c->D(DIVA_F_W_SURF_A); a.wb = c->D(DIVA_F_W_BASE_A);
  a.u3a = c->D(DIVA_F_U_3D_A); a.v3a = c->D(DIVA_F_V_3D_A);
  a.uva = c->D(DIVA_F_U_VAV_A); a.vva = c->D(DIVA_F_V_VAV_A); a.usa = c->D(DIVA_F_U_SURF_A);
  a.vsa = c->D(DIVA_F_V_SURF_A); a.uba = c->D(DIVA_F_U_BASE_A); a.vba = c->D(DIVA_F_V_BASE_A);
  a.abv = c->D(DIVA_F_UABS_VAV_A); a.abs_ = c->D(DIVA_F_UABS_SURF_A); a.abb = c->D(DIVA_F_UABS_BASE_A);
  a.Rs = c->D(DIVA_F_R_SHEAR);
  if (dyn != DIVA_DYN_SSA) k_secondary<true><<<G2>>>(a);
  else k_secondary<false><<<G2>>>(a);
  c->launches++;
  DIVA_LAUNCHED(c, "k_secondary");
  return DIVA_OK;
}

int launch_sia(Ctx* c) {
  k_sia<<<G2>>>(c->d, c->zt, c->c.n_flow, c->I(DIVA_F_MASK_SHEET_A), c->D(DIVA_F_HI_CX), c->D(DIVA_F_HI_CY),
                c->D(DIVA_F_DHS_DX_CX), c->D(DIVA_F_DHS_DY_CX), c->D(DIVA_F_DHS_DX_CY), c->D(DIVA_F_DHS_DY_CY),
                c->D(DIVA_F_A_FLOW_3D_CX), c->D(DIVA_F_A_FLOW_3D_CY), c->D(DIVA_F_U_3D_SIA_CX),
                c->D(DIVA_F_V_3D_SIA_CY)); c->launches++;
  DIVA_LAUNCHED(c, "k_sia");
  return DIVA_OK;
}

int launch_zero_velocities(Ctx* c, double* u, double* v) {
  k_zero_uv<<<G2>>>(c->d, u, v); c->launches++;
  DIVA_LAUNCHED(c, "k_zero_uv");
  return DIVA_OK;
}

int launch_any_sheet(Ctx* c, int* result) {
  int* flag = c->ff_flag;
  DIVA_CUDA(c, cudaMemsetAsync(flag, 0, sizeof(int), c->stream));
  k_count_sheet<<<G2>>>(c->d, c->I(DIVA_F_MASK_SHEET_A), flag); c->launches++;
  DIVA_LAUNCHED(c, "k_count_sheet");
  int h = 0;
  DIVA_CUDA(c, cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  DIVA_CUDA(c, cudaStreamSynchronize(c->stream));
  *result = h;
  return DIVA_OK;
}

}  // namespace diva
