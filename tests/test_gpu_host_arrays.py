"""Host arrays in and results out at the sizes where the way changes: small copies on the compute stream (64 KB), results in
page-locked blocks (64 KB to 16 MB, a few at a time), strided and zero-dimensional sources, results that outlive the next call."""
import numpy as np
import pytest

from b200.shlo.builder import Builder


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 16383, 16384, 16385, 300_001, (16 << 20) // 4, (16 << 20) // 4 + 1])
def test_round_trip(client, n):
    b = Builder()
    x = b.arg((n,), "f32")
    exe = client.compile(b.module([b.add(x, b.full((n,), 1.0, "f32"))]))
    src = np.arange(2 * n + 8, dtype=np.float32)
    kept = [exe(src[k:k + n])[0] for k in range(7)]            # more than the pool lends
    kept.append(exe(src[:2 * n:2])[0])
    for k in range(7):
        np.testing.assert_array_equal(kept[k], src[k:k + n] + 1)
        kept[k] += 1                                           # writable, and nobody else's
    np.testing.assert_array_equal(kept[7], src[:2 * n:2] + 1)
    np.testing.assert_array_equal(kept[0], src[:n] + 2)


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["f16", "f64", "i8", "ui16", "i64", "i1"])
def test_element_types(client, dt):
    np_t = {"f16": np.float16, "f64": np.float64, "i8": np.int8, "ui16": np.uint16, "i64": np.int64, "i1": np.bool_}[dt]
    x = (np.arange(40000).reshape(200, 200) % 2).astype(np_t)
    buf = client.buffer_from_host(x.T)
    assert buf.dtype == dt and buf.shape == (200, 200)
    np.testing.assert_array_equal(buf.to_numpy(), x.T)
    zero_d = client.buffer_from_host(np.array(1, np_t))
    assert zero_d.shape == () and zero_d.to_numpy() == np_t(1)
