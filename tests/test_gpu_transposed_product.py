"""Products that are only read transposed are made transposed: both layouts of both operands, 32 and 16 bits; a product that
something else reads too, or with a side too short for tiles, keeps its transpose. Held to float64 (K additions of rounded
products for f32, one rounding to 8 bits for bf16)."""
import numpy as np
import pytest

from b200.shlo.builder import Builder
from util import run_gpu


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["f32", "bf16"])
@pytest.mark.parametrize("lc,rc", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k,kept", [(200, 96, 64, ""), (17, 300, 40, ""), (128, 128, 128, "read"), (200, 8, 64, "short")])
def test_transposed_product(client, dt, lc, rc, m, n, k, kept):
    r = np.random.default_rng(m + n + 2 * lc + rc)
    a = (np.round(r.standard_normal((k, m) if lc == 0 else (m, k)) * 16) / 16).astype(np.float32)
    w = (np.round(r.standard_normal((k, n) if rc == 0 else (n, k)) * 16) / 16).astype(np.float32)
    b = Builder()
    y = b.dot_general(b.arg(a.shape, dt), b.arg(w.shape, dt), ((lc,), (rc,)))
    t = b.transpose(y, (1, 0))
    text = b.module([t, b.neg(y)] if kept == "read" else [t])
    assert ("transpose" in client.compile(text).plan_text()) == bool(kept)
    got, _ = run_gpu(client, text, [a, w], [dt, dt])
    want = (a.T if lc == 0 else a).astype(np.float64) @ (w if rc == 0 else w.T).astype(np.float64)
    tol = 1e-5 if dt == "f32" else 2.0 ** -8
    np.testing.assert_allclose(np.asarray(got[0], np.float64), want.T, rtol=tol, atol=tol * np.sqrt(k))
