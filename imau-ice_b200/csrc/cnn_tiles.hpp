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

}  // namespace diva::cnn
