"""fp32 products on the FMA pipe: both layouts of both operands, sizes around the tiles (32 x 64, 64 x 64, 64 x 128), k below
and above a stage, K splits over a cluster, groups, and rows that 16-byte copies cannot address."""
import numpy as np
import pytest

from b200.shlo.builder import Builder

SHAPES = [(1, 1, 3, 1), (31, 5, 63, 1), (32, 64, 64, 1), (33, 65, 65, 1), (64, 288, 1024, 1), (65, 130, 129, 1), (128, 260, 64, 3), (77, 77, 66, 6),
          (250, 784, 1000, 1), (462, 512, 512, 1), (2000, 96, 1500, 1), (20, 1000, 10, 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("m,k,n,g", SHAPES)
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_fma_product(client, monkeypatch, m, k, n, g, ta, tb):
    monkeypatch.setenv("B200_NO_TILE32", "1")          # the larger ones otherwise go to the tensor cores
    rng = np.random.default_rng(m + k + n)
    lead = (g,) if g > 1 else ()
    a = rng.standard_normal(lead + ((k, m) if ta else (m, k))).astype(np.float32)
    w = rng.standard_normal(lead + ((n, k) if tb else (k, n))).astype(np.float32)
    b = Builder()
    o = len(lead)
    y = b.dot_general(b.arg(a.shape, "f32"), b.arg(w.shape, "f32"), ((o + (0 if ta else 1),), (o + (1 if tb else 0),)), ((0,), (0,)) if g > 1 else ((), ()))
    exe = client.compile(b.module([y]))
    assert " fma tile=" in exe.plan_text(), exe.plan_text()
    got = exe(a, w)[0]
    want = np.matmul((a.swapaxes(-1, -2) if ta else a).astype(np.float64), (w.swapaxes(-1, -2) if tb else w).astype(np.float64))
    np.testing.assert_allclose(got, want, rtol=1e-5, atol=3e-6 * np.sqrt(k))
    np.testing.assert_array_equal(got, exe(a, w)[0])
