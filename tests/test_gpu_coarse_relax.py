"""The coarsest level relaxed by sweeps, where its matrix has no usable inverse: an ice cap without
basal friction (regularised Coulomb sliding at a till friction angle of zero).  Its twenty
viscosity iterations took 1038 V-cycles with the sweeps of the per-point kernels; as many, within a
tenth for the rounding, show sweeps of the same rows in the same order."""
import numpy as np
import pytest
import torch

from imau_ice_b200 import diva
import helpers

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU (B200)")]


@pytest.mark.parametrize("graphs", [True, False])
def test_sweeps_of_the_coarsest_level_precondition_as_before(monkeypatch, graphs):
    if not graphs:
        monkeypatch.setenv("DIVA_NO_GRAPHS", "1")
    g, cfg, f = helpers.make_case(2, dx=40e3, overrides={"choice_sliding_law": "Coulomb_regularised",
                                                         "picard_stop": "relres", "picard_relres_tol": 1e-6,
                                                         "DIVA_visc_it_nit": 20, "lin_adaptive": 1})
    ctx = diva.Context(g, cfg)
    helpers.prepare(ctx, f)
    r = ctx.solve_DIVA()
    assert r["picard_iterations"] == 20 and r["mg_cycles"] <= 1.1 * 1038, r
    assert np.isfinite(ctx.download(["u_vav_cx"])["u_vav_cx"]).all()
    ctx.close()
