"""The network's device-buffer forms on the caller's own buffers: outputs and targets at any
float's address give the same bits as on 16-byte boundaries, and nothing beside them is written."""
import threading

import numpy as np
import pytest
import torch

from imau_ice_b200 import _abi, diva, learned
import cnn_reference as ref
import helpers

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


def test_buffers_aligned_less_are_refused_before_any_launch():
    g = diva.Grid(9, 9, 10e3)
    net = learned.WarmStartNet(g, batch=1, capacity=0, seed=1)
    n = int(np.prod(net.padded_shape))
    feat = torch.zeros(n * learned.IN_C + 8, dtype=torch.bfloat16, device="cuda")
    out = torch.zeros(n * learned.N_OUT + 2, device="cuda")
    for df, do in ((2, 0), (8, 0), (0, 1), (0, 2)):
        for call in (lambda: net.forward(feat.data_ptr() + df, out.data_ptr() + do, 1),
                     lambda: net.train_step(feat.data_ptr() + df, out.data_ptr() + do, 1, 0.0)):
            with pytest.raises(diva.DivaError) as e:
                call()
            assert e.value.status == _abi.BAD_INPUT
    net.forward(feat.data_ptr(), out.data_ptr(), 1)
    net.close()


@pytest.mark.parametrize("ny, nx", [(2, 400), (4, 372), (3, 1001)])
def test_images_of_one_row_at_the_coarsest_level(ny, nx):
    """Forward pass and gradients of a strip four rows high (one at a quarter of the resolution)
    against the PyTorch reference, within the bounds of the network's other tests."""
    g = diva.Grid(nx, ny, 10e3)
    net = learned.WarmStartNet(g, batch=1, capacity=0, seed=nx)
    Hp, Wp = net.padded_shape
    rng = np.random.default_rng(nx)
    feat = torch.as_tensor(rng.normal(0, 1, (1, Hp, Wp, learned.IN_C))).to(torch.bfloat16)
    tgt = rng.normal(0, 1, (1, Hp, Wp, learned.N_OUT)).astype(np.float32)
    w = torch.as_tensor(net.get_weights()).requires_grad_(True)
    want = ref.forward(feat.float().numpy(), w, bf16=True)
    mask = np.broadcast_to(ref.valid_mask(Hp, Wp, ny, nx, g.nz), tgt.shape)
    ref.loss(want, torch.as_tensor(tgt), mask).backward()
    gref = w.grad.numpy()
    f, t = feat.cuda().contiguous(), torch.as_tensor(tgt).cuda()
    out = torch.zeros(1, Hp, Wp, learned.N_OUT, device="cuda")
    net.forward(f.data_ptr(), out.data_ptr(), 1)
    assert (out.cpu() - want.detach()).abs().max() < 2e-2 * want.detach().abs().max()
    net.train_step(f.data_ptr(), t.data_ptr(), 1, 0.0)
    gdev = net.grads()
    for name, (wo, shape, bo, nb) in learned.weight_layout()[0].items():
        m = int(np.prod(shape))
        for a, b, what in ((gdev[wo:wo + m], gref[wo:wo + m], "w"), (gdev[bo:bo + nb], gref[bo:bo + nb], "b")):
            assert np.linalg.norm(a - b) <= 5e-2 * max(np.linalg.norm(b), 1e-30), (name, what)
    net.close()


def test_networks_of_different_sizes_in_two_threads():
    """Each network trains from its own host thread; every call succeeds and the weights are those
    of the same training alone."""
    cases = []
    for dx in (200e3, 40e3):            # 9 x 15 and 41 x 71 cells
        g, cfg, f = helpers.make_case(2, dx=dx)
        ctx = diva.Context(g, cfg)
        helpers.prepare(ctx, f)
        net = learned.WarmStartNet(g, batch=1, capacity=8, seed=1)
        for _ in range(8):
            net.add_sample(ctx)
        ctx.close()
        w0 = net.get_weights()
        net.train(150, lr=1e-3, seed=2)
        cases.append((net, w0, net.get_weights()))
        net.set_weights(w0)
    failed = []

    def drive(net, w0, want):
        try:
            for _ in range(3):
                net.set_weights(w0)
                net.train(150, lr=1e-3, seed=2)
                if not np.array_equal(net.get_weights(), want):
                    failed.append("weights")
        except Exception as e:
            failed.append(e)
    threads = [threading.Thread(target=drive, args=c) for c in cases]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not failed, failed
    for c in cases:
        c[0].close()
