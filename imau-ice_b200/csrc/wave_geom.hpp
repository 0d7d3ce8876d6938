// Sizes of the streamed smoother (k_wave in solver.cu), the strips and chunks of a level, and
// whether it is swept in strips or smoothed by tiles, in plain C++ so that they can be checked for
// every level size without a GPU.
#pragma once
#include <cstddef>
#include "gpu.hpp"

namespace diva {

constexpr int kWavePre = 3;       // pairs of columns the copies run ahead
constexpr int kWaveBars = 8;      // mbarriers: more than the pairs in flight
constexpr int kWaveCopy = 5;      // copying warps: five of a pair's 20 plane columns each (a bulk copy takes about
                                  // 110 cycles to issue), the last the coarse columns
constexpr int kWaveCoarse = 8;    // coarse columns held (2 (kWavePre + 1) of a level not coarsened along i)
constexpr int kWaveSpin = 1 << 16;   // polls before a wait gives up: 0.26 s, a poll lasting up to 4 us (a copy
                                     // takes a few)

struct WaveGeom {
  static constexpr int NU = 2;   // sweeps per phase
  static constexpr int NP = 4 * NU, H = NP + 1;
  static constexpr int TJ = 64 - 2 * NP;              // largest tile height: pass 0's rows of a colour fill a warp
  static constexpr int HB = (H + 3) / 4 * 4;          // ring rows before the tile (even: 16-byte aligned)
  static constexpr int RP = (HB + TJ + H + 3) / 4 * 4;   // ring rows
  static constexpr int NC = 2 * kWavePre + 3 * NP + 6;   // ring columns: from the copies' to the output's left neighbour
  static constexpr int CP = RP + 8;                   // rows of a coarse column (a level not coarsened along j)
  static constexpr std::size_t xk = (std::size_t)NC * 8 * RP * sizeof(double), b = (std::size_t)NC * 2 * RP * sizeof(double);
  static constexpr std::size_t coarse = (std::size_t)kWaveCoarse * 2 * CP * sizeof(double);
  static constexpr std::size_t smem_down = xk + b + 128, smem_up = xk + b + coarse + 128;
  // two per pass (rows below and above the middle); output (descent: a warp per component, half
  // of the rows and column, ascent: per half of the rows); copies; prolongation (ascent: a lane
  // per row, component and column)
  static_assert(NC % 2 == 0 && (8 * RP * sizeof(double)) % 128 == 0 && (2 * RP) % 16 == 0, "pairs of slots, whole banks");
  static constexpr int passes = 2 * NP, out_down = 8, out_up = 2, pro = RP * 4 / 32;
  static constexpr int warps_down = passes + out_down + kWaveCopy, warps_up = passes + out_up + kWaveCopy + pro;
  static_assert(RP * 4 % 32 == 0 && warps_up <= 32 && warps_down <= 32, "warps of a block");
};

struct WaveShape {
  int rows, chunk;       // tile height and width
  int nstrip, nchunk;
  long steps;            // in turn on an SM
};
// Strips as high as two warps per pass allow (fewer halo rows), evened out over the level; then the
// number of chunks with the fewest steps in turn, each block (one per SM) taking half its chunk,
// halo and lag, and some to start, over as many rounds as needed.
inline WaveShape wave_shape(int ny, int nx) {
  using G = WaveGeom;
  WaveShape s{};
  const int ns = (ny + G::TJ - 1) / G::TJ;
  s.rows = ((ny + ns - 1) / ns + 1) / 2 * 2;
  s.nstrip = (ny + s.rows - 1) / s.rows;
  long best = 0;
  for (int n = 1; n <= nx; ++n) {
    const int w = (nx + n - 1) / n, nc = (nx + w - 1) / w;
    if (w < 4 && n > 1) break;
    const long rounds = ((long)s.nstrip * nc + kSMs - 1) / kSMs;
    const long cost = rounds * ((w + G::H + 3 * G::NP + 2) / 2 + 5);
    if (best == 0 || cost < best) {
      best = cost;
      s.chunk = w;
      s.nchunk = nc;
    }
  }
  s.steps = best;
  return s;
}

// Tiles of a level: 32 x 32 while that still fills the GPU, else 16 x 16, and 1.5x wider along i
// (T x 3T/2) when square tiles give a little more than one block per SM (e.g. 198 of 32 x 32 at
// 321 x 561, where 50 SMs would run two blocks each and set the kernel's length) and the wider
// ones fit in one block per SM, with less halo per point.
struct TileChoice {
  int edge;
  bool wide;
  long n;   // tiles
};
inline TileChoice tile_choice(int ny, int nx) {
  auto tiles = [&](int tj, int ti) { return (long)((ny + tj - 1) / tj) * ((nx + ti - 1) / ti); };
  TileChoice t{};
  t.edge = tiles(32, 32) >= kSMs ? 32 : 16;
  const long square = tiles(t.edge, t.edge), wide = tiles(t.edge, 3 * t.edge / 2);
  t.wide = square > kSMs && wide <= kSMs;
  t.n = t.wide ? wide : square;
  return t;
}

// Whether a level in double with two sweeps per phase is swept in strips: more points than one
// round of 16 x 16 tiles covers (two per SM), and no more steps in turn than the tiles take time
// for.  A smoothing pair takes 1.3 to 1.5 us a step.  Tiles take 33 us for one round of 16 x 16 ones
// and 46 to 60 for two, 49 to 53 for one of 32 x 48, and of 32 x 32 ones, two per SM, 50 to 59 us for
// one round, 70 to 105 for two and about 28 us for every 148 from there on.  Tiles against
// strips: 33.1 / 37.6 us at 201 x 351 (286 tiles of 16 x 16), 49.6 / 39.0 at 229 x 401 (390),
// 53.3 / 48.2 at 321 x 561 (126 of 32 x 48), 59.0 / 61.5 at 401 x 701 (286 of 32 x 32), 101 / 83 at
// 501 x 875 (448), 408 / 312 at 1501 x 1501 (2209); on long grids, whose strips are low or
// whose chunks are long, 47.2 / 64.7 at 6579 x 17, 50.1 / 63.6 at 49 x 4235, 82.8 / 102 at 41 x 8667,
// but 98.6 / 57.2 at 12198 x 41 and 92.6 / 62.8 at 6168 x 33.
inline bool strips_pay(int ny, int nx) {
  if ((long long)nx * ny < 2LL * kSMs * 16 * 16) return false;
  const TileChoice t = tile_choice(ny, nx);
  if (t.edge == 16) return true;
  const double per_sm = (double)t.n / kSMs;
  const double steps = t.wide ? 37.0 : per_sm <= 2.0 ? 40.0 : per_sm < 52.0 / 19.5 ? 52.0 : 19.5 * per_sm;
  return wave_shape(ny, nx).steps <= steps;
}

}  // namespace diva
