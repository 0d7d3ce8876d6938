"""The convolutions' choice of tiles (imau-ice_b200/csrc/cnn_tiles.hpp), compiled for the CPU and
checked for every layer over image sizes from one row or column on: the tiles cover the image,
their positions fit the accumulators, the launch's shared memory stays within what a block may
have, and no weight-gradient sum runs over more pixels than 64 slices of 64-pixel chunks gave, and
an eighth."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imau-ice_b200", "csrc")
LAYERS = [(16, 32), (32, 32), (32, 64), (64, 64), (64, 128), (128, 64), (64, 32)]
SIZES = [(1, w) for w in (*range(1, 300), 511, 1001)] + [(2, w) for w in range(1, 300, 7)] + \
        [(h, w) for h in (3, 5, 8, 21, 64, 141, 564) for w in (1, 2, 5, 16, 33, 81, 129, 324, 1001)]

PROGRAM = r"""
#include "cnn_tiles.hpp"
using namespace diva::cnn;
extern "C" void conv(int n, int H, int W, int KC, int NO, int* o) {
  const ConvTile t = conv_tile(n, H, W, KC, NO);
  const int v[] = {t.TW, t.TH, t.P, t.npx, t.ncol, t.nrow, t.ntile, conv_blocks(KC, NO), conv_smem(KC, NO, t.npx), kDynSmemMax};
  for (int k = 0; k < 10; ++k) o[k] = v[k];
}
extern "C" void wgrad(int n, int H, int W, int CI, int CO, int* o) {
  const WgradTile t = wgrad_tile(n, H, W, CI, CO);
  const int v[] = {t.TW, t.TH, t.zp, t.xp, t.ncol, t.nrow, t.ntile, t.buf, t.slices, kDynSmemMax};
  for (int k = 0; k < 10; ++k) o[k] = v[k];
}
"""


@pytest.fixture(scope="module")
def tiles(tmp_path_factory):
    d = tmp_path_factory.mktemp("tiles")
    (d / "t.cpp").write_text(PROGRAM)
    so = str(d / "t.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(d / "t.cpp"), "-o", so], check=True)
    return C.CDLL(so)


def ints(fn, *args, n):
    o = (C.c_int * n)()
    fn(*args, o)
    return list(o)


@pytest.mark.parametrize("cin, cout", LAYERS)
def test_convolution_tiles_cover_the_image_and_fit(tiles, cin, cout):
    for H, W in SIZES:
        for KC, NO in ((cin, cout), (cout, cin)):
            TW, TH, P, npx, ncol, nrow, ntile, nb, smem, limit = ints(tiles.conv, 2, H, W, KC, NO, n=10)
            assert TW >= 1 and TH >= 1 and P == TW + 2, (H, W, KC, NO)
            assert ncol * TW >= W and (ncol - 1) * TW < W and nrow * TH >= H and (nrow - 1) * TH < H
            assert ntile == 2 * ncol * nrow
            assert TH * P <= 128 * nb and (TH + 2) * P <= npx and 128 * nb - 1 + 2 * P + 2 < npx < 1 << 14
            assert smem <= limit <= 225 * 1024, (H, W, KC, NO, smem)


@pytest.mark.parametrize("cin, cout", LAYERS)
def test_weight_gradient_tiles_fit_and_keep_the_chains_short(tiles, cin, cout):
    for n in (1, 2, 8):
        for H, W in SIZES:
            TW, TH, zp, xp, ncol, nrow, ntile, buf, slices, limit = ints(tiles.wgrad, n, H, W, cin, cout, n=10)
            assert TW in (16, 32, 48, 64) and 1 <= TH <= 8
            assert ncol * TW >= W and nrow * TH >= H and ntile == n * ncol * nrow
            assert zp >= TW and xp >= TH * (TW + 2) and max(zp, xp) < 1 << 14
            zrow = cout // 8 * zp * 16
            assert buf >= (TH + 2) * zrow + max(cin // 8 * xp * 16, 128 // cout * zrow)
            assert 2 * buf + 128 <= limit
            assert 1 <= slices <= ntile
            chunks = -(-n * H * W // 64)
            before = 64 * -(-chunks // min(chunks, 64))     # chunks of the longest of up to 64 slices
            assert -(-ntile // slices) * min(TW, W) * TH <= before * 9 / 8, (n, H, W, slices)
