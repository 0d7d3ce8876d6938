"""DIVA_err after a solve that ends with a status: the field holds the last iteration that
reached its velocity update, 2 |u - u_prev| / |u + u_prev + 1e-5| (zero below the velocity
tolerance), also when no further iteration follows."""
import numpy as np
import pytest
import torch

from imau_ice_b200 import _abi, diva
import helpers

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU (B200)")]


@pytest.mark.parametrize("over, graphs", [
    # the first update overflows the squares of the second iteration's nonlinear residual
    ({"picard_stop": "relres", "DIVA_visc_it_relax": 1e146}, True),
    ({"picard_stop": "relres", "DIVA_visc_it_relax": 1e146}, False),
    # the first update overflows its own step norm
    ({"DIVA_visc_it_relax": 1e300}, True),
])
def test_a_solve_that_overflows_keeps_its_last_error_field(monkeypatch, over, graphs):
    if not graphs:
        monkeypatch.setenv("DIVA_NO_GRAPHS", "1")
    g, cfg, f = helpers.make_case(2, dx=40e3, overrides=over)
    ctx = diva.Context(g, cfg)
    helpers.prepare(ctx, f)
    with pytest.raises(diva.DivaError) as e:
        ctx.solve_DIVA()
    assert e.value.status == _abi.NAN_DETECTED
    o = ctx.download(["u_vav_cx", "v_vav_cy", "u_cx_prev", "v_cy_prev", "DIVA_err_cx", "DIVA_err_cy"])
    ctx.close()
    for u, up, err in (("u_vav_cx", "u_cx_prev", "DIVA_err_cx"), ("v_vav_cy", "v_cy_prev", "DIVA_err_cy")):
        un, uo = o[u], o[up]
        assert np.isfinite(un).all() and np.abs(un).max() > 1e100
        want = np.where(np.abs(un) > float(np.float32(1e-6)), 2.0 * np.abs(un - uo) / np.abs(un + uo + 1e-5), 0.0)
        np.testing.assert_allclose(o[err], want, rtol=1e-14, atol=0)
