"""The one-block sub-cycle, its set-up and the layer-grouped column kernels on the GPU at the sizes
where their splits go wrong: grids that are one or a few multigrid levels, levels with more rows
than the sub-cycle's threads hold, coarsening along one direction only, and layer counts that are
no multiple of the layers a thread takes.  Three viscosity iterations with linear solves to 1e-12
against the oracle's; both sides then differ by the solves' error times the systems' condition,
within the 1e-6 of the parity tests."""
import numpy as np
import pytest
import torch

import helpers
import oracle_backend as ob

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU (B200)")]


@pytest.mark.parametrize("cfg_id, dx, nz", [
    (2, 200e3, 3),     # 9 x 15
    (2, 90e3, 7),      # 17 x 31
    (2, 45e3, 5),      # 35 x 63: the sub-cycle from the finest level or the next
    (2, 33e3, 16),     # 49 x 85
    (1, 16e3, 4),      # 5 x 41: coarsened along the channel only
    (1, 3.3e3, 2),     # 25 x 193
])
def test_small_grids_and_layer_counts_match_the_oracle(cuda, oracle, cfg_id, dx, nz):
    g, cfg, f = helpers.make_case(cfg_id, dx=dx, overrides={"DIVA_visc_it_nit": 3, "lin_rtol": 1e-12},
                                  zeta=np.linspace(0.0, 1.0, nz))
    rg, og = helpers.run(cuda, g, cfg, f)
    ro, oo = helpers.run(oracle, g, cfg, f, oracle_solver=(ob.LIN_GMRES_WARM, 1e-12, 0.0))
    assert rg["picard_iterations"] == ro["picard_iterations"]
    for k in ("u_vav_cx", "v_vav_cy", "u_3D_cx", "v_3D_cy", "u_3D_a", "v_3D_a"):
        assert np.isfinite(og[k]).all()
        assert helpers.rel_l2(og[k], oo[k]) <= 1e-6, k
    assert helpers.rel_l2(og["w_3D_a"], oo["w_3D_a"]) <= 1e-5
    for k in ("A_flow_3D_cx", "A_flow_3D_cy", "A_flow_vav_a"):
        assert helpers.rel_l2(og[k], oo[k]) <= 1e-12, k
