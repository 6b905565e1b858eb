"""fp32 contractions by tiled copies: convolutions with their two gradients and dense products in every layout of A, at sizes
with ragged tiles, ragged K, K splits and several tiles per CTA."""
import numpy as np
import pytest
import torch

from b200.shlo.builder import Builder


def _product(client, m, k, n, ta, tb, g=1):
    rng = np.random.default_rng(m + k + n)
    lead = (g,) if g > 1 else ()
    a = rng.standard_normal(lead + ((k, m) if ta else (m, k))).astype(np.float32)
    w = rng.standard_normal(lead + ((n, k) if tb else (k, n))).astype(np.float32)
    b = Builder()
    o = len(lead)
    y = b.dot_general(b.arg(a.shape, "f32"), b.arg(w.shape, "f32"), ((o + (0 if ta else 1),), (o + (1 if tb else 0),)), ((0,), (0,)) if g > 1 else ((), ()))
    exe = client.compile(b.module([y]))
    assert " tile mode=" in exe.plan_text(), exe.plan_text()
    got = exe(a, w)[0]
    want = np.matmul((a.swapaxes(-1, -2) if ta else a).astype(np.float64), (w.swapaxes(-1, -2) if tb else w).astype(np.float64))
    np.testing.assert_allclose(got, want, rtol=1e-5, atol=1e-5 * np.abs(want).max())
    np.testing.assert_array_equal(got, exe(a, w)[0])


@pytest.mark.gpu
@pytest.mark.parametrize("m,k,n,ta,tb,g", [(462, 2048, 512, 0, 0, 1), (462, 2048, 512, 0, 1, 1), (1024, 1000, 1030, 0, 0, 1), (2048, 462, 1500, 1, 0, 1),
                                           (700, 1100, 4000, 1, 1, 1), (516, 900, 1999, 0, 1, 3), (512, 999, 8003, 1, 0, 1), (16384, 512, 130, 0, 0, 1)])
def test_dense_products(client, m, k, n, ta, tb, g):
    _product(client, m, k, n, ta, tb, g)


@pytest.mark.gpu
@pytest.mark.parametrize("batch,size,cin,cout", [(8, 32, 64, 64), (5, 16, 96, 128), (16, 8, 128, 256), (13, 4, 256, 512), (3, 32, 32, 200)])
@pytest.mark.parametrize("ksize", [3, 1])
def test_convolution_and_its_gradients(client, batch, size, cin, cout, ksize):
    rng = np.random.default_rng(batch)
    x = rng.standard_normal((batch, size, size, cin)).astype(np.float32)
    w = (rng.standard_normal((ksize, ksize, cin, cout)) / np.sqrt(ksize * ksize * cin)).astype(np.float32)
    up = rng.standard_normal((batch, size, size, cout)).astype(np.float32)
    b = Builder()
    xv, wv, uv = b.arg(x.shape, "f32"), b.arg(w.shape, "f32"), b.arg(up.shape, "f32")
    pad = ((ksize // 2, ksize // 2),) * 2
    y = b.conv(xv, wv, padding=pad)
    grads = b.grad(b.reduce_sum(b.mul(y, uv), (0, 1, 2, 3)), [xv, wv])
    exe = client.compile(b.module([y, *grads]))
    if ksize == 3 and batch >= 8:
        assert " tile mode=1" in exe.plan_text(), exe.plan_text()
    got = exe(x, w, up)
    tx = torch.tensor(x, dtype=torch.float64).permute(0, 3, 1, 2).requires_grad_()
    tw = torch.tensor(w, dtype=torch.float64).permute(3, 2, 0, 1).requires_grad_()
    ty = torch.nn.functional.conv2d(tx, tw, padding=ksize // 2)
    (ty * torch.tensor(up, dtype=torch.float64).permute(0, 3, 1, 2)).sum().backward()
    for g, want in zip(got, (ty.permute(0, 2, 3, 1), tx.grad.permute(0, 2, 3, 1), tw.grad.permute(2, 3, 1, 0))):
        want = want.detach().numpy()
        np.testing.assert_allclose(g, want, rtol=1e-5, atol=1e-5 * np.abs(want).max())
