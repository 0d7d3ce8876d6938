"""The shapes of the smoother without a GPU: the strips and chunks of a level
(imau-ice_b200/csrc/wave_geom.hpp, compiled for the CPU) cover it within the kernel's limits; the
streamed schedule restated in test_wave_schedule gives the colour sweeps at the heights that
choice makes, those of two more than a multiple of four among them; and the autotuner times
the strips beside the square tiles."""
import ctypes as C
import inspect
import os
import random
import subprocess

import numpy as np
import pytest

from imau_ice_b200 import autotune, diva
import test_wave_schedule as ws

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imau-ice_b200", "csrc")
PROGRAM = r"""
#include "wave_geom.hpp"
using namespace diva;
extern "C" void shape(int ny, int nx, int* o) {
  const WaveShape s = wave_shape(ny, nx);
  const int v[] = {s.rows, s.chunk, s.nstrip, s.nchunk, WaveGeom::TJ};
  for (int k = 0; k < 5; ++k) o[k] = v[k];
}
extern "C" void choice(int ny, int nx, int* o) {
  const TileChoice t = tile_choice(ny, nx);
  const int v[] = {t.edge, t.wide, (int)t.n, (int)strips_pay(ny, nx)};
  for (int k = 0; k < 4; ++k) o[k] = v[k];
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("wave")
    (d / "w.cpp").write_text(PROGRAM)
    so = str(d / "w.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(d / "w.cpp"), "-o", so], check=True)
    return C.CDLL(so)


@pytest.fixture(scope="module")
def shape(lib):
    def call(ny, nx):
        o = (C.c_int * 5)()
        lib.shape(ny, nx, o)
        return list(o)
    return call


# ny, nx: the default tiles (edge, wide), and whether strips take the smoothing pair less time there
@pytest.mark.parametrize("ny, nx, tiles, strips", [
    (351, 201, (16, 0), 0), (401, 229, (16, 0), 1), (561, 321, (32, 1), 1), (701, 401, (32, 0), 0), (875, 501, (32, 0), 1),
    (1501, 1501, (32, 0), 1), (9, 5005, (32, 1), 0), (9, 8710, (32, 0), 0), (8710, 9, (32, 0), 0), (17, 6579, (32, 1), 0),
    (25, 8106, (32, 0), 0), (33, 2570, (32, 1), 1), (33, 6168, (32, 0), 1), (49, 4235, (32, 0), 0), (4235, 49, (32, 0), 0),
    (65, 3078, (32, 0), 0), (3078, 65, (32, 0), 1), (8667, 41, (32, 0), 0), (41, 8667, (32, 0), 1), (113, 2691, (32, 0), 1),
    (4485, 113, (32, 0), 0), (129, 4100, (32, 0), 1), (4100, 129, (32, 0), 0), (1025, 129, (32, 1), 1)])
def test_the_faster_smoother_is_the_default(lib, ny, nx, tiles, strips):
    o = (C.c_int * 4)()
    lib.choice(ny, nx, o)
    assert (o[0], o[1]) == tiles and o[3] == strips


def test_strips_and_chunks_cover_every_level(shape):
    seen = set()
    for ny in (*range(5, 200), 211, 321, 501, 999, 1501, 20000):
        for nx in (5, 9, 50, 211, 561, 1501, 16001):
            rows, chunk, nstrip, nchunk, top = shape(ny, nx)
            assert 2 <= rows <= top == 48 and rows % 2 == 0 and chunk >= 4
            assert nstrip * rows >= ny and (nstrip - 1) * rows < ny
            assert nchunk * chunk >= nx and (nchunk - 1) * chunk < nx and nchunk < 65536
            seen.add(rows % 4)
    assert seen == {0, 2}


@pytest.mark.parametrize("nx, ny, chunk", [(13, 6, 13), (12, 49, 7), (10, 53, 4)])
def test_schedule_at_the_chosen_heights(shape, nx, ny, chunk):
    rows = shape(ny, nx)[0]
    # the restatement's own bound is on multiples of four; nothing else in it depends on that
    src = inspect.getsource(ws.wave)
    assert "rows % 4 == 0" in src
    scope = dict(vars(ws))
    exec(src.replace("rows % 4 == 0", "rows % 2 == 0"), scope)
    rng, order = np.random.default_rng(ny), random.Random(nx)
    L = ws.Level(nx, ny, ws.SIDES[2])
    co, b = rng.normal(0, 0.3, (18, 9)), rng.normal(0, 1, (2, ny, nx))
    x = np.zeros((2, ny, nx))
    for _ in range(2):
        for p in range(4):
            ws.colour_pass(L, x, b, co, p >> 1, p & 1)
    got, _ = scope["wave"](L, None, b, co, 2, rows, chunk, False, rng=order)
    K = ws.Level((nx + 2) // 2, (ny + 2) // 2, ws.SIDES[2])
    xc = rng.normal(0, 1, (2, K.ny, K.nx))

    def coarse(cp, Cj, Ci):
        lj, li = (K.ny - 1, K.nx - 2) if cp == 0 else (K.ny - 2, K.nx - 1)
        q = K.src(cp, min(max(Cj, 0), lj), min(max(Ci, 0), li))
        return 0.0 if q is None else xc[cp][q]
    y = x.copy()
    inner = np.array([[[L.interior(c, j, i) for i in range(nx)] for j in range(ny)] for c in (0, 1)])
    for c, j, i in zip(*np.nonzero(inner)):
        y[c, j, i] += ws.prolong(K, c, j, i, 2, 2, coarse)
    for _ in range(2):
        for p in (3, 2, 1, 0):
            ws.colour_pass(L, y, b, co, p >> 1, p & 1)
    up, _ = scope["wave"](L, got, b, co, 2, rows, chunk, True, K, xc, 2, 2, rng=order)
    assert np.array_equal(got[inner], x[inner]) and np.array_equal(up[inner], y[inner])


class StripCtx:
    """A level swept in strips by default (1.5 ms) above a tiled one: edge 16 takes 1 ms, 32 2 ms."""

    def __init__(self, strip_ms=1.5):
        self.grid = diva.Grid(321, 561, 5e3)
        self.cfg = type("Cfg", (), {"precision": 0, "choice_ice_margin": 0})()
        self.edges, self.strip_ms = [], strip_ms

    def nonlinear_residual(self):
        return 0.0

    def set_tile_edges(self, e):
        self.edges = list(e)

    def get_tile_edges(self):
        e = (self.edges + [0] * 3)[:3]
        return [e[0] or 32, e[1] or 16, 0]

    def get_strip_rows(self):
        return [0 if self.edges and self.edges[0] else 46, 0, 0]

    def profile_kernel(self, which, reps):
        e = (self.edges + [0] * 3)[:3]
        return {0: self.strip_ms, 16: 2.5, 32: 2.0}[e[0]] + {0: 9.0, 16: 1.0, 32: 2.0}[e[1]], 0.0


@pytest.mark.parametrize("strip_ms, want", [(1.5, [0, 16, 0]), (3.0, [32, 16, 0])])
def test_tuner_keeps_the_strips_where_they_are_fastest(tmp_path, strip_ms, want):
    assert len(list(autotune.candidates([32, 16, 0], [46, 0, 0]))) == 6
    cache = str(tmp_path / "tiles.json")
    ctx = StripCtx(strip_ms)
    edges, t = autotune.tune_tile_edges(ctx, reps=1, trials=1, cache=cache)
    assert ctx.edges == want and len(t) == 6 and edges == [32, 16, 0]
    again = StripCtx(strip_ms)
    assert autotune.tune_tile_edges(again, cache=cache) == (edges, {}) and again.edges == want
