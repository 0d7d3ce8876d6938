"""The convolution kernels at the image sizes where their tiles are ragged: forward pass and
gradients against the PyTorch reference with the device's BF16 roundings, within the bounds of
the network's other tests."""
import numpy as np
import pytest
import torch

from imau_ice_b200 import diva, learned
import cnn_reference as ref

pytestmark = pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU (B200)")


@pytest.mark.gpu
@pytest.mark.parametrize("ny,nx,n", [(5, 5, 1), (8, 130, 3), (131, 9, 1), (64, 60, 2)])
def test_forward_and_gradients_at_ragged_sizes(ny, nx, n):
    g = diva.Grid(nx, ny, 10e3)
    net = learned.WarmStartNet(g, batch=n, capacity=0, seed=ny + nx)
    Hp, Wp = net.padded_shape
    rng = np.random.default_rng(ny)
    feat = rng.normal(0, 1, (n, Hp, Wp, learned.IN_C)).astype(np.float32)
    feat = torch.as_tensor(feat).to(torch.bfloat16).float().numpy()
    tgt = rng.normal(0, 1, (n, Hp, Wp, learned.N_OUT)).astype(np.float32)
    w = torch.as_tensor(net.get_weights()).requires_grad_(True)
    want = ref.forward(feat, w, bf16=True)
    mask = np.broadcast_to(ref.valid_mask(Hp, Wp, ny, nx, g.nz), tgt.shape)
    ref.loss(want, torch.as_tensor(tgt), mask).backward()
    gref = w.grad.numpy()
    f = torch.as_tensor(feat).to(torch.bfloat16).cuda().contiguous()
    t = torch.as_tensor(tgt).cuda().contiguous()
    out = torch.zeros(n, Hp, Wp, learned.N_OUT, device="cuda")
    net.forward(f.data_ptr(), out.data_ptr(), n)
    assert (out.cpu() - want.detach()).abs().max() < 2e-2 * want.detach().abs().max()
    net.train_step(f.data_ptr(), t.data_ptr(), n, 0.0)
    gdev = net.grads()
    for name, (wo, shape, bo, nb) in learned.weight_layout()[0].items():
        m = int(np.prod(shape))
        for a, b, what in ((gdev[wo:wo + m], gref[wo:wo + m], "w"), (gdev[bo:bo + nb], gref[bo:bo + nb], "b")):
            assert np.linalg.norm(a - b) <= 5e-2 * max(np.linalg.norm(b), 1e-30), (name, what)
    net.close()
