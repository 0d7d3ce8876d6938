"""Square tiles that the caller chose, on double levels below and above the size from which the
default sweeps in strips, and the wide tiles of long narrow grids: each gives the per-colour
kernels' solve bit for bit."""
import numpy as np
import pytest
import torch

from imau_ice_b200 import diva
import helpers

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU (B200)")]
FRONT = {"choice_ice_margin": "BC"}


def long_channel(times, dx=10e3, across=False):
    """A channel (65 x 9 cells at 10 km) with every column repeated, along i or along j."""
    g, cfg, f = helpers.make_case(1, dx=dx)
    nx, ny = g.nx * times, g.ny
    f = {k: np.repeat(v, times, axis=-1) for k, v in f.items()}
    if across:
        nx, ny, f = ny, nx, {k: np.swapaxes(v, -1, -2) for k, v in f.items()}
    return diva.Grid(nx, ny, g.dx, zeta=g.zeta), cfg, f


@pytest.mark.parametrize("case, over, edge, strips", [
    (dict(cfg_id=2, dx=10e3), {}, 32, False),                          # 161 x 281
    (dict(cfg_id=2, dx=8.3e3), {}, 32, False),                         # 193 x 337, just below the limit
    (dict(cfg_id=1, dx=1.9e3, calving_front=True), FRONT, 32, False),  # 337 x 43, 'BC' front rows
    (dict(cfg_id=2, dx=6.7e3), {}, 32, True),                          # 239 x 417
    (dict(cfg_id=2, dx=6.7e3), {}, 16, True),
    (dict(cfg_id=1, dx=0.75e3, calving_front=True), FRONT, 32, True),  # 853 x 107
    (dict(times=77), {}, None, False),                                 # 5005 x 9: 32 x 48 tiles
    (dict(times=77), {}, 32, False),
    (dict(times=36, dx=5e3), {}, None, True),                          # 4644 x 17: one strip of 18 rows
    (dict(times=36, dx=5e3, across=True), {}, None, True),             # 17 x 4644: chunks as wide as the level
])
def test_shapes_match_per_colour_kernels(monkeypatch, case, over, edge, strips):
    g, cfg, f = long_channel(**case) if "times" in case else helpers.make_case(**case)
    cfg = dict(cfg, **over, DIVA_visc_it_nit=4, lin_rtol=1e-4)
    out = []
    for tiles in (True, False):
        if not tiles:
            monkeypatch.setenv("DIVA_NO_TILES", "1")
        ctx = diva.Context(g, cfg)
        helpers.prepare(ctx, f)
        if tiles:
            edges = ctx.get_tile_edges()
            assert edges[0] != 0 and (ctx.get_strip_rows()[0] != 0) == strips
            if edge:
                ctx.set_tile_edges([edge] * len(edges))
                assert ctx.get_tile_edges()[0] == edge and not any(ctx.get_strip_rows())
            else:
                assert edges[0] == (16 if strips else 32)
        else:
            assert not any(ctx.get_tile_edges()) and not any(ctx.get_strip_rows())
        r = ctx.solve_DIVA()
        out.append((r, ctx.download(["u_vav_cx", "v_vav_cy"])))
        ctx.close()
    (ra, oa), (rb, ob) = out
    assert ra["status"] == rb["status"] and ra["mg_cycles"] == rb["mg_cycles"] > 0
    for k in oa:
        assert np.array_equal(oa[k], ob[k]), k
        assert np.isfinite(oa[k]).all() and np.abs(oa[k]).max() > 1.0
