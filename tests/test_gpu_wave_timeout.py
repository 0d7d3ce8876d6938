"""Failure detection of the streamed smoother, without a GPU fault: with DIVA_WAVE_DROP=1 it
issues no copies, so that every block's wait runs out after its quarter of a second.  The kernels
end by themselves, the graph-launched and the host-driven solve and the timing entry return
TIMEOUT after few V-cycles, and the GPU and the context stay usable."""
import numpy as np
import pytest
import torch

from imau_ice_b200 import _abi, diva
import helpers

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU (B200)")]


def case():
    return helpers.make_case(2, dx=7.1e3, overrides={"DIVA_visc_it_nit": 3, "lin_rtol": 1e-4})   # 225 x 395


@pytest.mark.parametrize("graphs", [True, False])
def test_a_wait_that_runs_out_fails_the_solve(monkeypatch, graphs):
    if not graphs:
        monkeypatch.setenv("DIVA_NO_GRAPHS", "1")
    g, cfg, f = case()
    ok = diva.Context(g, cfg)
    helpers.prepare(ok, f)
    want = ok.solve_DIVA()
    u = ok.download(["u_vav_cx"])["u_vav_cx"]
    ok.close()
    monkeypatch.setenv("DIVA_WAVE_DROP", "1")
    ctx = diva.Context(g, cfg)
    monkeypatch.delenv("DIVA_WAVE_DROP")
    helpers.prepare(ctx, f)
    n0 = ctx.kernel_launches()
    for what in (ctx.solve_DIVA, lambda: ctx.profile_kernel(3, 1), ctx.solve_DIVA):   # again: nothing sticks
        with pytest.raises(diva.DivaError) as e:
            what()
        assert e.value.status == _abi.TIMEOUT and "did not arrive" in str(e.value)
    assert ctx.kernel_launches() - n0 < 400          # a V-cycle or two each, not the iteration limit
    ctx.profile_kernel(2, 1)                         # kernels that wait for nothing succeed
    ctx.close()
    after = diva.Context(g, cfg)
    helpers.prepare(after, f)
    r = after.solve_DIVA()
    assert r["mg_cycles"] == want["mg_cycles"]
    assert np.array_equal(after.download(["u_vav_cx"])["u_vav_cx"], u)
    after.close()
