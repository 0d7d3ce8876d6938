// common.cuh -- layout, constants and helpers shared by the B200 kernels.
//
// Device layout.  Every 2D field (a, cx, cy and b grid alike) lives on one
// padded plane of nx columns x ld rows, element (j,i) at [i*ld + j] with j
// fastest -- the order of the reference's Fortran arrays (ny,nx), so a warp
// over j reads 32 consecutive doubles.  A cx field uses columns 0..nx-2, a
// cy field rows 0..ny-2, a b field both.  3D fields are layer-major:
// (k,j,i) at [k*plane + i*ld + j], so each zeta layer is one coalesced plane.
// ld is ny rounded up to 16 elements (128-byte rows for doubles).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "../../include/diva.h"
#include "gpu.hpp"

namespace diva {

// parameters_module.f90:10-23
constexpr double kPi = 3.141592653589793;
constexpr double kT0 = 273.16;
constexpr double kCC = 8.7E-04;
constexpr double kGrav = 9.81;
constexpr double kRhoI = 910.0;
constexpr double kRhoSW = 1028.0;
constexpr double kRGas = 8.314;
// DIVA_vel_tolerance = 1e-6 is a default-REAL literal in ice_velocity_module.f90:1547
constexpr double kVelTol = (double)1e-6f;

constexpr int kMaxNz = 64;

struct Dims {
  int nx, ny, nz, ld;
  long long plane;  // nx * ld
  double dx;
  __host__ __device__ long long at(int j, int i) const { return (long long)i * ld + j; }
};

// zeta tables passed by value to kernels
struct Zeta {
  int nz;
  double z[kMaxNz];    // C%zeta
  double z2[kMaxNz];   // zeta**2 (computed on the host with pow, as the reference's zeta**n)
  double zn[kMaxNz];   // zeta**n_flow
};

// MAX and MIN as gfortran expands them for the reference (mvar = a; if (b > mvar
// .OR. isnan(mvar)) mvar = b): a NaN argument never wins.  Written out with an
// explicit NaN test so that the result does not depend on how min/max
// instructions are selected for NaN operands.
__host__ __device__ __forceinline__ double max_ref(double a, double b) { return (b > a || a != a) ? b : a; }
__host__ __device__ __forceinline__ double min_ref(double a, double b) { return (b < a || a != a) ? b : a; }

__device__ __forceinline__ double stag_margin(double v0, double v1, double H0, double H1) {
  // calc_staggered_margin, ice_velocity_module.f90:1300-1319
  if (H0 > 0.0 && H1 == 0.0) return v0;
  if (H0 == 0.0 && H1 > 0.0) return v1;
  return 0.5 * (v0 + v1);
}

// 2D launch helpers: threadIdx.x -> j (coalesced), threadIdx.y / blockIdx.y -> i
constexpr int kBX = 32, kBY = 8;
inline dim3 grid2d(int nj, int ni) { return dim3((nj + kBX - 1) / kBX, (ni + kBY - 1) / kBY); }
inline dim3 block2d() { return dim3(kBX, kBY); }
// Kernels over 3D fields.  A thread loads kLayers layers of its column before it uses or stores
// any: a loop that loads, computes and stores layer by layer waits for memory once per layer,
// the compiler not being able to move a load over a store.  Where the layers are independent
// the grid has a block per kLayers of them (grid_layers), which also fills the GPU on small grids.
// 1001 x 1001 x 15: staggering of one field 82 -> 58 us, k_secondary 688 -> 260 us, SIA velocities
// 157 -> 95 us, rate factor 71 -> 60 us; staggering on 161 x 281 15.2 -> 4.9 us.
constexpr int kLayers = 5;
inline dim3 grid_layers(int nj, int ni, int nz) {
  dim3 g = grid2d(nj, ni);
  g.z = (nz + kLayers - 1) / kLayers;
  return g;
}
// (loads: of the last layer again instead of behind a branch, where there are fewer left)
#define FOR_LAYERS(e, k0, nz) _Pragma("unroll") for (int e = 0; e < kLayers; ++e) if ((k0) + e < (nz))
#define LOAD_LAYERS(e, k, k0, nz)                      \
  _Pragma("unroll") for (int e = 0; e < kLayers; ++e)  \
    if (const int k = (k0) + e < (nz) ? (k0) + e : (nz) - 1; true)

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide sum of up to 4 values; result valid in thread 0.  blockDim <= 1024.
template <int N>
__device__ __forceinline__ void block_sum(double (&v)[N]) {
  __shared__ double sh[N][32];
  const int lane = (threadIdx.x + threadIdx.y * blockDim.x) & 31;
  const int warp = (threadIdx.x + threadIdx.y * blockDim.x) >> 5;
  const int nwarp = (blockDim.x * blockDim.y + 31) >> 5;
#pragma unroll
  for (int q = 0; q < N; ++q) v[q] = warp_sum(v[q]);
  __syncthreads();
  if (lane == 0) {
#pragma unroll
    for (int q = 0; q < N; ++q) sh[q][warp] = v[q];
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int q = 0; q < N; ++q) {
      double t = lane < nwarp ? sh[q][lane] : 0.0;
      v[q] = warp_sum(t);
    }
  }
}

// ---- reductions finished by the kernel that starts them ---------------------------------
// Blocks of 32 x 8 threads walk the points in 32 (j) x 8 (i) tiles, tile t, t + gridDim.x, ...;
// at most kRedBlocks of them (the four that k_matvec's registers let an SM hold: with six a second
// round starts half empty), so that the last block's sum over the blocks' partials stays at a
// few microseconds (one partial per tile: 23 us at 1501 x 1501).
constexpr int kRedBlocks = 4 * kSMs;
inline int red_blocks(const Dims& d) {
  const int n = ((d.ny + kBX - 1) / kBX) * ((d.nx + kBY - 1) / kBY);
  return n < kRedBlocks ? n : kRedBlocks;
}
#define FOR_TILES(d)                                                                                  \
  for (int nbx_ = ((d).ny + kBX - 1) / kBX, nt_ = nbx_ * (((d).nx + kBY - 1) / kBY), t_ = blockIdx.x; \
       t_ < nt_; t_ += gridDim.x)                                                                     \
    if (const int j = (t_ % nbx_) * kBX + threadIdx.x, i = (t_ / nbx_) * kBY + threadIdx.y;           \
        j < (d).ny && i < (d).nx)

struct Reduction {
  double* partials;   // the blocks' sums
  int* count;         // blocks that have stored theirs: zero before and after every kernel
};
// The grid's sum of v: true in thread 0 of the block that finishes last, which has the totals
// (block sums added in block order by a fixed tree: the same bits whichever block is last).
template <int N>
__device__ __forceinline__ bool reduce_all(double (&v)[N], const Reduction& red) {
  __shared__ bool last;
  const int t = threadIdx.x + threadIdx.y * blockDim.x, nt = blockDim.x * blockDim.y;
  block_sum<N>(v);
  if (t == 0) {
#pragma unroll
    for (int q = 0; q < N; ++q) __stcg(red.partials + (long long)N * blockIdx.x + q, v[q]);
    __threadfence();
    last = atomicAdd(red.count, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
#pragma unroll
  for (int q = 0; q < N; ++q) v[q] = 0.0;
  for (int b = t; b < (int)gridDim.x; b += nt)
#pragma unroll
    for (int q = 0; q < N; ++q) v[q] += __ldcg(red.partials + (long long)N * b + q);
  block_sum<N>(v);
  if (t == 0) *red.count = 0;
  return t == 0;
}

}  // namespace diva
