// The tiles of the convolution kernels (cnn.cu): sizes and choice, in plain C++ so that they can
// be checked for every image size without a GPU.
#pragma once
#include <algorithm>

namespace diva::cnn {

// Dynamic shared memory a convolution kernel may ask for: an SM's 227 KB per block less 2 KB for
// what the kernels declare themselves.
constexpr int kDynSmemMax = 225 * 1024;

// Planes of 16-byte chunks are `px` pixels long; a warp stores chunks c8 = 0.. of one or more
// consecutive pixels, so px is rounded up to the residue mod 8 that puts those 8 stores of a
// phase into different banks (C = 16: 2 chunks x 4 pixels, 32: 4 x 2, 64 and more: 8 x 1).
constexpr int plane_px(int px, int C) {
  const int r = C == 16 ? 4 : C == 32 ? 2 : 1;
  return px + ((r - px % 8) + 8) % 8;
}

// ---- forward / dgrad: a tile is TH x TW output pixels; its input, with the halo, is staged as
// (TH + 2) rows of P = TW + 2 pixels
struct ConvTile {
  int TW, TH, P, npx;   // npx: pixels of a staged plane
  int ncol, nrow, ntile;
};
// accumulator blocks per tile: two where the weights leave room for two or more CTAs per SM
constexpr int conv_blocks(int KC, int NO) { return KC * NO <= 64 * 32 ? 2 : 1; }
// bytes between the 8-channel planes of one tap's weights (padded like plane_px), and of all taps
constexpr int conv_wplane(int KC, int NO) { return plane_px(NO, KC) * 16; }
constexpr int conv_wbytes(int KC, int NO) { return 9 * (KC / 8) * conv_wplane(KC, NO); }
constexpr int conv_smem(int KC, int NO, int npx) { return conv_wbytes(KC, NO) + (KC / 8) * npx * 16 + 128; }

// The tile of a forward / dgrad convolution of n H x W images: of all column splits whose tile fits
// in shared memory (images of one row would take the widest: 250 KB at 128 -> 64 channels) the
// one with the least work, counting the accumulator rows (128 per block, the halo columns and
// the ragged ends among them) and the staged pixels of all tiles.
inline ConvTile conv_tile(int n, int H, int W, int KC, int NO) {
  ConvTile best{};
  double cost = 0.0;
  const int rows = 128 * conv_blocks(KC, NO);
  for (int ncol = 1; ncol <= W; ++ncol) {
    const int TW = (W + ncol - 1) / ncol, P = TW + 2, npx = plane_px(rows + 2 * P + 2, KC);
    if ((W + TW - 1) / TW != ncol || P > rows || conv_smem(KC, NO, npx) > kDynSmemMax) continue;
    if (best.TW && TW < 8) break;
    const int TH = std::min(H, rows / P), nrow = (H + TH - 1) / TH;
    const double c = (double)ncol * nrow * (rows + (TH + 2) * P);
    if (!best.TW || c < cost) {
      cost = c;
      best = ConvTile{TW, TH, P, npx, ncol, nrow, n * ncol * nrow};
    }
  }
  return best;
}

// ---- weight gradient: a tile is TH rows of X (TW + 2 pixels, halo columns included) and the
// TH + 2 rows of dZ (TW pixels) that they meet
struct WgradTile {
  int TW, TH, zp, xp;   // zp: pixels between dZ chunk groups; xp: of an X plane
  int ncol, nrow, ntile;
  int buf;              // bytes of one of the two tile buffers
  int slices;           // the tiles are dealt to, each with its own sums
};
// The longest chain of additions to one accumulator, in pixels.  The tensor core truncates every
// addition to its FP32 accumulator, so a sum shrinks with the length of its chain: with 64
// slices of whole 64-pixel chunks it would be `chain` pixels; tiles, whose ragged ends count
// whole here, may make it an eighth longer (4 % on 8 samples of 321 x 561: an error of 1.77e-5
// against a sum known in 64 bits, as with the chunks).
inline long wgrad_chain(int n, int H, int W) {
  const long chunks = ((long)n * H * W + 63) / 64, chain = (chunks + 63) / 64 * 64;
  return chain + chain / 8;
}
// The tile of a weight gradient: a multiple of 16 pixels wide (zeros beyond the image), the width
// with the fewest staged pixels; rows so that two tile buffers take about 110 KB at most (two
// CTAs per SM) and a tile is no longer than a chain.
inline WgradTile wgrad_tile(int n, int H, int W, int CI, int CO) {
  WgradTile t{};
  long cost = 0;
  for (int TW = 16; TW <= 64; TW += 16) {
    const long c = (long)((W + TW - 1) / TW) * (TW * CO + (TW + 2) * CI);
    if (!t.TW || c <= cost) {
      cost = c;
      t.TW = TW;
    }
  }
  const long chain = wgrad_chain(n, H, W);
  auto pixels = [&] { return (long)std::min(t.TW, W) * t.TH; };   // of the image in a tile
  t.zp = plane_px(t.TW, CO);
  for (t.TH = std::min(H, 8);; --t.TH) {
    t.xp = plane_px(t.TH * (t.TW + 2), CI);
    // dZ, then X; the last A operands run one or more dZ rows on (rows of D that nothing reads)
    const int zrow = CO / 8 * t.zp * 16, xbytes = CI / 8 * t.xp * 16;
    t.buf = ((t.TH + 2) * zrow + std::max(xbytes, 128 / CO * zrow) + 127) / 128 * 128;
    if ((2 * t.buf <= 110 * 1024 || t.TH <= 2) && (pixels() <= chain || t.TH == 1)) break;
  }
  t.ncol = (W + t.TW - 1) / t.TW;
  t.nrow = (H + t.TH - 1) / t.TH;
  t.ntile = n * t.ncol * t.nrow;
  // 64 slices (or a tile each), more where their chains were too long; a chain holds a tile at least
  t.slices = std::min(t.ntile, 64);
  if ((t.ntile + t.slices - 1) / t.slices * pixels() > chain) {
    const int each = (int)(chain / pixels());
    t.slices = (t.ntile + each - 1) / each;
  }
  return t;
}
inline long wgrad_part_floats(const WgradTile& t, int CI, int CO) { return (long)t.slices * (9L * CI * CO + CO); }

}  // namespace diva::cnn
