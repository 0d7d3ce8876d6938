// Sizes of the streamed smoother (k_wave in solver.cu) and the strips and chunks of a level, in
// plain C++ so that they can be checked for every level size without a GPU.
#pragma once
#include <cstddef>

namespace diva {

constexpr int kSMs = 148;   // B200

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
  return s;
}

}  // namespace diva
