"""The tile layout of the convolution kernels (imau-ice_b200/csrc/cnn.cu), restated on the
CPU: the staged tiles, read back through the canonical no-swizzle layouts that the matrix
descriptors describe, must give the forward convolution, its input gradient and its weight
gradient, at image sizes with ragged tiles, and every address must lie in the shared memory
the launch asks for.  K-major (in 16-byte units): ((8,m),2):((1,SBO),LBO); MN-major: chunk
groups SBO apart, 8 K rows of 16 bytes each, K groups LBO apart."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F


def plane_px(px, C):
    r = {16: 4, 32: 2}.get(C, 1)
    return px + (r - px % 8) % 8


def conv_tile(n, H, W, nb, C):
    best, cost = None, 0.0
    for ncol in range(1, W + 1):
        TW = -(-W // ncol)
        P = TW + 2
        if -(-W // TW) != ncol or P > 128 * nb:
            continue
        if best and TW < 8:
            break
        TH = min(H, 128 * nb // P)
        nrow = -(-H // TH)
        c = ncol * nrow * (128 * nb + (TH + 2) * P)
        if best is None or c < cost:
            best, cost = (TW, TH, P, plane_px(128 * nb + 2 * P + 2, C), ncol, nrow, n * ncol * nrow), c
    return best


def conv_kernel(x, w, KC, NO, dgrad):
    """k_conv3x3 without bias and ReLU: x [n][H][W][KC], w [9][NO][KC]; every D row of every
    tile is formed, the unstaged pixels hold NaN (they may reach dropped rows only)."""
    n, H, W, _ = x.shape
    nb, C8 = (2 if KC * NO <= 64 * 32 else 1), KC // 8
    TW, TH, P, npx, ncol, nrow, ntile = conv_tile(n, H, W, nb, KC)
    y = np.full((n, H, W, NO), np.nan, np.float32)
    for tile in range(ntile):
        c, q = tile % ncol, tile // ncol
        x0, y0, b = c * TW, (q % nrow) * TH, q // nrow
        sm = np.full((C8 * npx, 8), np.nan, np.float32)              # 16-byte chunks
        for p in range((TH + 2) * P):
            yy, xx = y0 - 1 + p // P, x0 - 1 + p % P
            v = x[b, yy, xx] if 0 <= yy < H and 0 <= xx < W else np.zeros(KC, np.float32)
            sm[np.arange(C8) * npx + p] = v.reshape(C8, 8)
        for blk in range(nb):
            D = np.zeros((128, NO), np.float32)
            for t in range(9):
                tt = 8 - t if dgrad else t
                a0 = blk * 128 + (tt // 3) * P + tt % 3
                rows = np.arange(128)
                for k8 in range(C8):                                   # SBO 128 B = 8 chunks, LBO = npx chunks
                    at = a0 + k8 * npx + rows
                    assert at.max() < C8 * npx
                    D += sm[at] @ w[t][:, k8 * 8:k8 * 8 + 8].T
            for m in range(128):
                py, px = divmod(blk * 128 + m, P)
                if py < TH and px < TW and y0 + py < H and x0 + px < W:
                    y[b, y0 + py, x0 + px] = D[m]
    return y


def wgrad_tile(n, H, W, CI, CO):
    TW, cost = 0, 0
    for tw in (16, 32, 48, 64):
        c = -(-W // tw) * (tw * CO + (tw + 2) * CI)
        if not TW or c <= cost:
            TW, cost = tw, c
    TH, zrow = min(H, 8), CO // 8 * plane_px(TW, CO) * 16
    while TH > 2 and 2 * (((TH + 2) * zrow + max(CI // 8 * plane_px(TH * (TW + 2), CI) * 16, 128 // CO * zrow) + 127)
                          // 128 * 128) > 110 * 1024:
        TH -= 1
    return TW, TH, plane_px(TW, CO), plane_px(TH * (TW + 2), CI), -(-W // TW), -(-H // TH)


def wgrad_kernel(x, dz, CI, CO):
    n, H, W, _ = x.shape
    I8, O8, NT = CI // 8, CO // 8, 128 // CO
    sets = {32: 1, 64: 2, 128: 3}[CO]
    TW, TH, zp, xp, ncol, nrow = wgrad_tile(n, H, W, CI, CO)
    XW = TW + 2
    zsize = (TH + 2) * O8 * zp
    total = zsize + max(I8 * xp, NT * O8 * zp)
    g = np.zeros((9, CO, CI), np.float32)
    gb = np.zeros(CO, np.float32)
    with np.errstate(invalid="ignore"):
        for tile in range(n * ncol * nrow):
            c, q = tile % ncol, tile // ncol
            x0, y0, b = c * TW, (q % nrow) * TH, q // nrow
            sm = np.full((total, 8), np.nan, np.float32)
            for p in range((TH + 2) * TW):
                r, xx = divmod(p, TW)
                yy = y0 - 1 + r
                v = dz[b, yy, x0 + xx] if 0 <= yy < H and x0 + xx < W else np.zeros(CO, np.float32)
                sm[(r * O8 + np.arange(O8)) * zp + xx] = v.reshape(O8, 8)
                if 1 <= r <= TH:
                    gb += v
            for p in range(TH * XW):
                yy, xx = y0 + p // XW, x0 - 1 + p % XW
                v = x[b, yy, xx] if yy < H and 0 <= xx < W else np.zeros(CI, np.float32)
                sm[zsize + np.arange(I8) * xp + p] = v.reshape(I8, 8)
            for r in range(TH):
                for xs in range(0, TW, 16):
                    kk = np.arange(16)
                    for s in range(sets):
                        za = (r + s * NT) * O8 * zp + xs
                        at = za + np.arange(16)[:, None] * zp + kk[None, :]       # [chunk group][k]
                        assert at.max() < total
                        A = sm[at].transpose(0, 2, 1).reshape(128, 16)             # [m][k]
                        for dx in range(3):
                            bt = zsize + r * XW + xs + dx + np.arange(I8)[:, None] * xp + kk[None, :]
                            assert bt.max() < total
                            B = sm[bt].transpose(0, 2, 1).reshape(CI, 16)
                            D = A @ B.T
                            for i in range(NT):
                                dyi = s * NT + i
                                if dyi < 3:
                                    g[3 * (2 - dyi) + dx] += D[i * CO:(i + 1) * CO]
    return g, gb


def reference(x, dz, w, CI, CO):
    """Forward, input gradient and weight gradient by autograd: w [9][CO][CI]."""
    xt = torch.as_tensor(x).permute(0, 3, 1, 2).double().requires_grad_(True)
    wt = torch.as_tensor(w).permute(1, 2, 0).reshape(CO, CI, 3, 3).double().requires_grad_(True)
    y = F.conv2d(xt, wt, padding=1)
    y.backward(torch.as_tensor(dz).permute(0, 3, 1, 2).double())
    return (y.detach().permute(0, 2, 3, 1).numpy(), xt.grad.permute(0, 2, 3, 1).numpy(),
            wt.grad.reshape(CO, CI, 9).permute(2, 0, 1).numpy())


@pytest.mark.parametrize("CI,CO", [(16, 32), (32, 32), (32, 64), (64, 128), (128, 64)])
@pytest.mark.parametrize("H,W", [(1, 1), (9, 21), (20, 7)])
def test_tiles_give_the_convolution_and_its_gradients(CI, CO, H, W):
    rng = np.random.default_rng(CI + CO + H)
    x, dz = (rng.normal(0, 1, (2, H, W, c)).astype(np.float32) for c in (CI, CO))
    w = rng.normal(0, 1, (9, CO, CI)).astype(np.float32)
    y, gx, gw = reference(x, dz, w, CI, CO)
    tol = 1e-5                       # FP32 sums of at most 9 x 128 terms against FP64
    np.testing.assert_allclose(conv_kernel(x, w, CI, CO, False), y, rtol=0, atol=tol * np.abs(y).max() * 10)
    if CI >= 32:
        got = conv_kernel(dz, np.ascontiguousarray(w.transpose(0, 2, 1)), CO, CI, True)
        np.testing.assert_allclose(got, gx, rtol=0, atol=tol * np.abs(gx).max() * 10)
    g, gb = wgrad_kernel(x, dz, CI, CO)
    np.testing.assert_allclose(g, gw, rtol=0, atol=tol * np.abs(gw).max() * 10)
    np.testing.assert_allclose(gb, dz.sum((0, 1, 2)), rtol=0, atol=1e-4)


@pytest.mark.parametrize("n,H,W", [(1, 564, 324), (8, 141, 81), (3, 2, 400), (1, 400, 2), (2, 63, 129),
                                   (1, 64, 64), (1, 128, 256)])
def test_tile_choice_covers_the_image_within_the_shared_memory(n, H, W):
    for KC, NO in [(16, 32), (32, 32), (32, 64), (64, 32), (64, 64), (64, 128), (128, 64)]:
        nb = 2 if KC * NO <= 64 * 32 else 1
        TW, TH, P, npx, ncol, nrow, ntile = conv_tile(n, H, W, nb, KC)
        assert ncol * TW >= W and nrow * TH >= H and ntile == n * ncol * nrow
        assert TH * P <= 128 * nb and (TH + 2) * P <= npx and 128 * nb - 1 + 2 * P + 2 < npx
        smem = 9 * (KC // 8) * plane_px(NO, KC) * 16 + (KC // 8) * npx * 16 + 128
        assert smem <= 227 * 1024
        CI, CO = KC, NO
        TW, TH, zp, xp, ncol, nrow = wgrad_tile(n, H, W, CI, CO)
        assert ncol * TW >= W and nrow * TH >= H and xp >= TH * (TW + 2) and zp >= TW
        zrow = CO // 8 * zp * 16
        buf = (TH + 2) * zrow + max(CI // 8 * xp * 16, 128 // CO * zrow)
        assert 2 * (buf + 128) + 128 <= 227 * 1024                # two tile buffers
        assert max(zp, xp) < 1 << 14 and npx < 1 << 14          # descriptor offsets, 14 bits of 16 bytes
