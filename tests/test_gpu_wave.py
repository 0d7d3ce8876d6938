"""Streamed smoothing of the large levels on the GPU: levels just above its size, ragged strips
and chunks, narrow and long grids, every kind of side, 'BC' front rows and the 16-row strips
give the per-colour kernels' solve bit for bit."""
import numpy as np
import pytest
import torch

from imau_ice_b200 import diva
import helpers

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU (B200)")]
FLIP = {f"BC_{c}_{s}": k for c, s, k in (("u", "west", "infinite"), ("u", "east", "zero"), ("u", "south", "zero"),
                                         ("u", "north", "infinite"), ("v", "west", "infinite"), ("v", "east", "zero"),
                                         ("v", "south", "infinite"), ("v", "north", "zero"))}


@pytest.mark.parametrize("cfg_id, dx, over, gen, edge", [
    (2, 7.6e3, {}, {}, None),                                          # 211 x 369: just above the limit
    (2, 7.1e3, FLIP, {}, None),                                        # 225 x 395
    (2, 6.7e3, {}, {}, 16),                                            # 239 x 417 in 16-row strips
    (1, 0.75e3, {}, {}, None),                                         # 107 x 853: three strips
    (1, 0.75e3, {"choice_ice_margin": "BC"}, {"calving_front": True}, None),
    (1, 0.75e3, dict(FLIP, choice_ice_margin="BC"), {"calving_front": True}, 16),
])
def test_streamed_levels_match_per_colour_kernels(monkeypatch, cfg_id, dx, over, gen, edge):
    g, cfg, f = helpers.make_case(cfg_id, dx=dx, overrides=dict(over, DIVA_visc_it_nit=4, lin_rtol=1e-4), **gen)
    out = []
    for tiles in (True, False):
        if not tiles:
            monkeypatch.setenv("DIVA_NO_TILES", "1")
        ctx = diva.Context(g, cfg)
        helpers.prepare(ctx, f)
        if tiles:
            n = len(ctx.get_tile_edges())
            assert ctx.get_tile_edges()[0] != 0
            if edge:
                ctx.set_tile_edges([edge] * n)
        r = ctx.solve_DIVA()
        out.append((r, ctx.download(["u_vav_cx", "v_vav_cy"])))
        ctx.close()
    (ra, oa), (rb, ob) = out
    assert ra["status"] == rb["status"] and ra["mg_cycles"] == rb["mg_cycles"] > 0
    for k in oa:
        assert np.array_equal(oa[k], ob[k]), k
        assert np.isfinite(oa[k]).all() and np.abs(oa[k]).max() > 1.0
