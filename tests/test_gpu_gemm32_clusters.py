"""fp32 products on the FMA pipe whose K eight CTAs of a cluster share: part rows of a tile, part columns, the last CTA's k short
or missing, both layouts of both operands (tolerance as for the other splits: K additions of rounded products)."""
import numpy as np
import pytest

from b200.shlo.builder import Builder


@pytest.mark.gpu
@pytest.mark.parametrize("m,k,n", [(31, 1024, 250), (20, 1000, 200), (120, 4096, 65), (64, 1024, 288), (33, 901, 130), (1, 1100, 251)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_cluster_of_eight(client, monkeypatch, m, k, n, ta, tb):
    monkeypatch.setenv("B200_NO_TILE32", "1")
    rng = np.random.default_rng(m + k + n)
    a = rng.standard_normal((k, m) if ta else (m, k)).astype(np.float32)
    w = rng.standard_normal((n, k) if tb else (k, n)).astype(np.float32)
    b = Builder()
    exe = client.compile(b.module([b.dot_general(b.arg(a.shape, "f32"), b.arg(w.shape, "f32"), ((0 if ta else 1,), (1 if tb else 0,)))]))
    assert "cluster=8" in exe.plan_text(), exe.plan_text()
    got = exe(a, w)[0]
    want = (a.T if ta else a).astype(np.float64) @ (w.T if tb else w).astype(np.float64)
    np.testing.assert_allclose(got, want, rtol=1e-5, atol=3e-6 * np.sqrt(k))
    np.testing.assert_array_equal(got, exe(a, w)[0])
