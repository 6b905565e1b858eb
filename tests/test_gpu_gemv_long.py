"""One row times a matrix whose columns are contiguous and long (K from 8192 to 16384, where a block's warps share a column):
ragged K, fewer columns than blocks, several columns per block, both 16-bit types."""
import numpy as np
import pytest
import torch

from b200.shlo.builder import Builder


@pytest.mark.gpu
@pytest.mark.parametrize("k,n", [(8192, 2048), (8200, 300), (12296, 1), (16384, 1777), (16376, 9472)])
@pytest.mark.parametrize("dt", ["bf16", "f16"])
def test_one_row(client, k, n, dt):
    gen = torch.Generator().manual_seed(k)
    t = {"bf16": torch.bfloat16, "f16": torch.float16}[dt]
    x = torch.randn(1, k, generator=gen).to(t)
    w = torch.randn(n, k, generator=gen).to(t)
    b = Builder()
    y = b.dot_general(b.convert(b.arg((1, k), "f32"), dt), b.convert(b.arg((n, k), "f32"), dt), ((1,), (1,)), out_dtype="f32")
    got = client.compile(b.module([y]))(x.float().numpy(), w.float().numpy())[0]
    want = (x.double() @ w.double().T).numpy()
    np.testing.assert_allclose(got, want, rtol=1e-4, atol=2e-3)
