"""The viscosity of a column's layers, one layer a thread on small grids and three on large ones,
against the oracle: sizes on either side of the change and layer counts that leave none, one or
two layers for the last thread.  The bound is that of the state completion's other test."""
import numpy as np
import pytest
import torch

from imau_ice_b200 import diva
import helpers

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU (B200)")]


@pytest.mark.parametrize("dx, nz, margin", [
    (10e3, 16, "infinite_slab"),   # 161 x 281: six groups of layers are fewer than the GPU's threads
    (9e3, 16, "infinite_slab"),    # 177 x 311: more, the last group of one layer
    (9e3, 17, "BC"),               # of two
    (8e3, 15, "BC"),               # 201 x 351: of three
    (9e3, 7, "infinite_slab"),     # three groups: one layer a thread
    (60e3, 2, "BC"),
])
def test_layers_match_the_oracle(cuda, oracle, dx, nz, margin):
    g, cfg, f = helpers.make_case(2, dx=dx, overrides={"choice_ice_margin": margin}, zeta=np.linspace(0.0, 1.0, nz) ** 0.8)
    rng = np.random.default_rng(nz)
    x, y = np.meshgrid(np.linspace(-1, 1, g.nx), np.linspace(-1, 1, g.ny))
    uv = {"u_vav_cx": np.asfortranarray(80.0 * x[:, :-1] + rng.normal(0, 3, (g.ny, g.nx - 1))),
          "v_vav_cy": np.asfortranarray(50.0 * y[:-1] + rng.normal(0, 3, (g.ny - 1, g.nx)))}
    names = ["visc_eff_3D_a", "visc_eff_int_a", "beta_eff_a", "du_dz_3D_cx", "dv_dz_3D_cy", "taub_cx"]
    out = []
    for be in (cuda, oracle):
        ctx = diva.Context(g, cfg, be)
        helpers.prepare(ctx, f)
        ctx.upload(uv)
        ctx.complete_state(3)
        out.append(ctx.download(names))
        ctx.close()
    for k in names:
        assert np.isfinite(out[0][k]).all() and np.abs(out[0][k]).max() > 0.0, k
        assert helpers.rel_l2(out[0][k], out[1][k]) <= 1e-9, k
