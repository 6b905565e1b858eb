"""The radix form of stablehlo.sort and the selecting form of chlo.top_k at the sizes where they change over: one tile and
one element more, rows that are no multiple of a warp's 256, candidates that overflow, k at its limits."""
import numpy as np
import pytest

from b200.shlo.builder import Builder
from oracle import interp
from util import run_gpu


def _keys(shape, dt, seed=3, spread=50):
    rng = np.random.default_rng(seed)
    if dt in ("f32", "bf16"):
        x = (np.round(rng.standard_normal(shape) * spread) / 8).astype(np.float32)
        x.reshape(-1)[[0, 2, 5, 9]] = [np.nan, -0.0, 0.0, -np.inf]
        return x
    return rng.integers(0 if dt[0] == "u" else -spread, spread, shape).astype({"i32": np.int32, "ui32": np.uint32, "ui8": np.uint8}[dt])


@pytest.mark.gpu
@pytest.mark.parametrize("shape,dt", [((3, 127), "f32"), ((3, 128), "f32"), ((2, 300), "ui32"), ((2, 4096), "f32"), ((4, 4097), "f32"),
                                      ((2, 8192), "i32"), ((3, 30522), "f32"), ((1, 64001), "ui32")])
@pytest.mark.parametrize("descending", [False, True])
def test_radix_sort(client, shape, dt, descending):
    x = _keys(shape, dt)
    tag = np.arange(x.size, dtype=np.int32).reshape(shape)
    half = (np.arange(x.size) % 7).astype(np.int16).reshape(shape)
    b = Builder()
    text = b.module(b.sort([b.arg(shape, "i16"), b.arg(shape, dt), b.arg(shape, "i32")], 1, comparator=lambda s, a0, b0, a1, b1, a2, b2: s.compare(
        a1, b1, "GT" if descending else "LT", "TOTALORDER" if dt == "f32" else None)))
    got, _ = run_gpu(client, text, [half, x, tag])
    want = interp.run_text(text, [half, x, tag])
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)


@pytest.mark.gpu
@pytest.mark.parametrize("shape,k,dt,spread", [((3, 511), 5, "f32", 50), ((3, 512), 128, "f32", 50), ((2, 2047), 100, "bf16", 50), ((2, 2048), 256, "f32", 4000),
                                               ((2, 8192), 512, "f32", 4000), ((2, 32769), 1, "i32", 1 << 30), ((3, 40000), 64, "f32", 2), ((2, 30522), 50, "ui8", 200)])
def test_selecting_top_k(client, shape, k, dt, spread):
    x = _keys(shape, dt, spread=spread)
    b = Builder()
    text = b.module(b.top_k(b.arg(shape, dt), k))
    got, _ = run_gpu(client, text, [x], dtypes=[dt])
    want = interp.run_text(text, [x])
    for g, w in zip(got, want):
        np.testing.assert_array_equal(np.asarray(g, np.float64), np.asarray(w, np.float64))


@pytest.mark.gpu
@pytest.mark.parametrize("fill", [np.nan, 1.5])
def test_top_k_of_equal_values_keeps_positions(client, fill):
    x = np.full((2, 5000), fill, np.float32)
    b = Builder()
    got, _ = run_gpu(client, b.module(b.top_k(b.arg(x.shape, "f32"), 9)), [x])
    np.testing.assert_array_equal(got[1], np.tile(np.arange(9, dtype=np.int32), (2, 1)))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1 << 22, (1 << 22) + 1])
def test_sort_at_the_longest_radix_row(client, n):
    x = np.random.default_rng(n).integers(-1000, 1000, (1, n)).astype(np.int32)
    b = Builder()
    text = b.module(b.sort([b.arg(x.shape, "i32"), b.iota(x.shape, "i32", 1)], 1, comparator=lambda s, a0, b0, a1, b1: s.compare(a0, b0, "LT")))
    got, _ = run_gpu(client, text, [x])
    order = np.argsort(x, axis=1, kind="stable").astype(np.int32)
    np.testing.assert_array_equal(got[1], order)
    np.testing.assert_array_equal(got[0], np.take_along_axis(x, order, 1))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1 << 18, (1 << 18) + 1])
def test_top_k_at_the_longest_row_of_a_block(client, n):
    x = np.random.default_rng(n).integers(-1000, 1000, (1, n)).astype(np.float32)
    b = Builder()
    got, _ = run_gpu(client, b.module(b.top_k(b.arg(x.shape, "f32"), 200)), [x])
    order = np.argsort(-x, axis=1, kind="stable")[:, :200].astype(np.int32)
    np.testing.assert_array_equal(got[1], order)
    np.testing.assert_array_equal(got[0], np.take_along_axis(x, order, 1))
