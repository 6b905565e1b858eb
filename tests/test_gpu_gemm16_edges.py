"""16-bit products whose result rows start on 16 bytes, on 4 bytes and on 2 bytes, with ragged last tiles, several tiles per
block, a K split and every result type."""
import numpy as np
import pytest
import torch

from b200.shlo.builder import Builder

TYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


@pytest.mark.gpu
@pytest.mark.parametrize("m,k,n", [(129, 72, 264), (300, 200, 518), (257, 64, 1003), (4000, 128, 2050), (130, 4096, 67), (31, 640, 33)])
@pytest.mark.parametrize("dt,out", [("bf16", "bf16"), ("f16", "f16"), ("bf16", "f32")])
def test_result_rows(client, m, k, n, dt, out):
    gen = torch.Generator().manual_seed(m + n)
    x = torch.randn(m, k, generator=gen).to(TYPES[dt])
    w = torch.randn(n, k, generator=gen).to(TYPES[dt])
    b = Builder()
    y = b.dot_general(b.convert(b.arg((m, k), "f32"), dt), b.convert(b.arg((n, k), "f32"), dt), ((1,), (1,)), ((), ()), **({"out_dtype": out} if out != dt else {}))
    exe = client.compile(b.module([b.convert(y, "f32")]))
    got = exe(x.float().numpy(), w.float().numpy())[0]
    want = (x.double() @ w.double().T).to(TYPES[out]).double().numpy()
    np.testing.assert_allclose(got, want, rtol=1e-2 if out != "f32" else 1e-4, atol=2e-2 if out != "f32" else 1e-3)
