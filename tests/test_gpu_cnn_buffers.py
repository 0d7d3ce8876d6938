"""The network's device-buffer forms on the caller's own buffers: outputs and targets at any
float's address give the same bits as on 16-byte boundaries, and nothing beside them is written."""
import numpy as np
import pytest
import torch

from imau_ice_b200 import diva, learned

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU (B200)")]


@pytest.mark.parametrize("shift", [1, 2, 3])
def test_outputs_and_targets_at_any_float(shift):
    g = diva.Grid(37, 29, 10e3)
    net = learned.WarmStartNet(g, batch=2, capacity=0, seed=3)
    shape = (2,) + net.padded_shape
    rng = np.random.default_rng(shift)
    feat = torch.as_tensor(rng.normal(0, 1, shape + (learned.IN_C,))).to(torch.bfloat16).cuda()
    tgt = torch.as_tensor(rng.normal(0, 1, shape + (learned.N_OUT,))).float().cuda()
    n = tgt.numel()
    res = []
    for at in (0, shift):
        out = torch.full((n + 8,), -7.0, device="cuda")
        t = torch.zeros(n + 8, device="cuda")
        t[at:at + n] = tgt.flatten()
        net.forward(feat.data_ptr(), out.data_ptr() + 4 * at, 2)
        loss = net.train_step(feat.data_ptr(), t.data_ptr() + 4 * at, 2, 0.0)
        out = out.cpu()
        assert (out[:at] == -7.0).all() and (out[at + n:] == -7.0).all()
        res.append((out[at:at + n].numpy(), net.grads(), loss))
    net.close()
    (o0, g0, l0), (o1, g1, l1) = res
    assert np.array_equal(o0, o1) and np.array_equal(g0, g1) and l0 == l1
