"""Gathers from a table that is a pointwise result: computed where they are used when they take at most a sixteenth of it,
read from memory otherwise, with indices at and beyond both ends."""
import numpy as np
import pytest

from b200.shlo.builder import Builder


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(1, 16), (3, 15), (7, 16), (33, 1001)])
@pytest.mark.parametrize("read_again", [False, True])
def test_labels_of_a_pointwise_table(client, rows, cols, read_again):
    rng = np.random.default_rng(rows + cols)
    x, bias = rng.standard_normal((rows, cols)).astype(np.float32), rng.standard_normal(cols).astype(np.float32)
    idx = rng.integers(0, cols, rows).astype(np.int32)
    idx[0], idx[-1] = -5, cols + 3
    b = Builder()
    t = b.sub(b.arg(x.shape, "f32"), b.broadcast_in_dim(b.arg((cols,), "f32"), x.shape, (1,)))
    y = b.take_along_last(t, b.arg((rows,), "i32"))
    z = b.take_rows(t, b.const_array(np.array([rows + 1, 0], np.int32)))
    got = client.compile(b.module([y, z] + ([b.exp(t)] if read_again else [])))(x, bias, idx)
    want = x - bias
    np.testing.assert_array_equal(got[0], want[np.arange(rows), np.clip(idx, 0, cols - 1)])
    np.testing.assert_array_equal(got[1], want[[rows - 1, 0]])
    if read_again:
        np.testing.assert_allclose(got[2], np.exp(want), rtol=1e-6)
