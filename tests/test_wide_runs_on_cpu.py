"""Threads that take several consecutive elements: where a run of four or eight stays in one aligned piece through slices,
pads, concatenations, transposes, broadcasts, windows and gathers it is read as one, where it does not each element is read by
itself. Random chains of such operations over extents on both sides of the multiples of four and eight, large enough for the
wide form, and row kernels and reductions over rows of such lengths, run on the CPU and held to the interpreter."""
import shutil

import numpy as np
import pytest

if shutil.which("g++") is None:
    pytest.skip("needs g++ to build the generated kernels for the host", allow_module_level=True)

from b200.shlo.builder import Builder
from cuda_emu import run_plan_on_cpu
from oracle import interp


def _check(text, inputs, tol):
    for g, w in zip(run_plan_on_cpu(text, inputs), interp.run_text(text, inputs), strict=True):
        w = np.asarray(w)
        assert g.shape == w.shape
        if g.dtype.kind in "iub":
            np.testing.assert_array_equal(g, w.astype(g.dtype))
        else:
            np.testing.assert_allclose(g.astype(np.float64), w.astype(np.float64), rtol=tol, atol=tol, equal_nan=True)


def chain(seed):
    """Up to five indexing operations on a small tensor, spread over 151 552 elements and more at the end by a broadcast, whose
    innermost dimension is the chain's own innermost or another one."""
    r = np.random.default_rng(seed)
    dt = str(r.choice(["f32", "bf16", "bf16", "i32"]))
    ext = [4, 8, 12, 16, 24, 8, 16, 6, 10, 3]
    shape = tuple(int(r.choice(ext)) for _ in range(int(r.integers(2, 4))))
    b = Builder()
    x = b.arg(shape, dt)
    inputs = [r.integers(-20, 20, shape).astype(np.int32) if dt == "i32" else (np.round(r.standard_normal(shape) * 8) / 8).astype(np.float32)]
    for _ in range(int(r.integers(1, 6))):
        k, rank = int(r.integers(0, 9)), x.ndim
        grid = int(r.choice([1, 4, 8]))
        if k == 0:
            x = b.transpose(x, tuple(int(v) for v in r.permutation(rank)))
        elif k == 1:
            x = b.reverse(x, [int(r.integers(0, rank))])
        elif k == 2:
            lo = [int(r.integers(0, s)) // grid * grid for s in x.shape]
            x = b.slice(x, lo, list(x.shape), [int(r.choice([1, 1, 1, 2])) for _ in x.shape])
        elif k == 3:
            lo, hi = ([int(r.integers(-1, 2)) * grid for _ in x.shape] for _ in range(2))
            if all(s + a + c > 0 for s, a, c in zip(x.shape, lo, hi)):
                x = b.pad(x, b.const(3 if dt == "i32" else 0.5, dt), lo, hi, [int(r.choice([0, 0, 0, 1])) if s + a + c < 30 and a >= 0 and c >= 0 else 0
                                                                                 for s, a, c in zip(x.shape, lo, hi)])
        elif k == 4 and x.size < 4096:
            d = int(r.integers(0, rank))
            y = b.slice(x, [0] * rank, [max(1, s // 2 // grid * grid) if i == d else s for i, s in enumerate(x.shape)])
            x = b.concatenate([x, y, x], d)
        elif k == 5:
            n = x.size
            f = int(r.choice([f for f in range(1, n + 1) if n % f == 0]))
            x = b.reshape(x, (f, n // f))
        elif k == 6:
            idx = b.arg((8,), "i32")
            inputs.append(r.integers(-2, x.shape[0] + 2, 8).astype(np.int32))
            x = b.take_rows(b.reshape(x, (x.shape[0], x.size // x.shape[0])), idx)
        elif k == 7:
            d = int(r.integers(0, rank))
            s = b.arg((), "i32")
            inputs.append(np.array(int(r.integers(-2, x.shape[d] + 2)), np.int32))
            at = [s if i == d else b.const(0, "i32") for i in range(rank)]
            if r.random() < 0.5:
                x = b.dynamic_slice(x, at, tuple(max(1, v // 2) if i == d else v for i, v in enumerate(x.shape)))
            else:
                u = b.slice(x, [0] * rank, [max(1, v // 2) if i == d else v for i, v in enumerate(x.shape)])
                x = b.dynamic_update_slice(x, b.neg(u), at)
        elif k == 8:
            x = b.add(x, x)
    lead = -(-151552 // x.size)
    lead += -lead % 8
    inner = r.random() < 0.75
    full = (lead, *x.shape) if inner else (*x.shape, lead)
    y = b.broadcast_in_dim(x, full, tuple(range(1, x.ndim + 1)) if inner else tuple(range(x.ndim)))
    other = b.arg((full[-1],), dt)
    inputs.append(r.integers(-5, 5, full[-1]).astype(np.int32) if dt == "i32" else (np.round(r.standard_normal(full[-1]) * 8) / 8).astype(np.float32))
    return b.module([b.add(y, b.broadcast_in_dim(other, full, (len(full) - 1,)))]), inputs


@pytest.mark.parametrize("seed", range(12))
def test_wide_pointwise_kernels(seed):
    text, inputs = chain(seed)
    _check(text, inputs, 2e-2 if "bf16" in text else 1e-5)


@pytest.mark.parametrize("rows,n,dt", [(1300, 128, "bf16"), (1190, 96, "f32"), (1184, 70, "bf16"), (3, 1032, "bf16"), (9, 512, "f32"), (2, 8200, "bf16"), (5, 2049, "f32")])
def test_rows_in_registers(rows, n, dt):
    """A layer norm with a bias in front: whole and partial rounds of a warp's and a block's row, kept in registers or not."""
    r = np.random.default_rng(n)
    b = Builder()
    x, bias, scale = b.arg((rows, n), dt), b.arg((n,), dt), b.arg((n,), "f32")
    y = b.add(x, b.bcast(bias, x.shape, (1,)))
    y = b.convert(y, "f32") if dt != "f32" else y
    c = b.sub(y, b.bcast(b.mean(y, (1,)), y.shape, (0,)))
    inv = b.rsqrt(b.add(b.mean(b.mul(c, c), (1,)), b.full((rows,), 1e-5, "f32")))
    z = b.mul(b.mul(c, b.bcast(inv, y.shape, (0,))), b.bcast(scale, y.shape, (1,)))
    inputs = [(np.round(r.standard_normal(s) * 8) / 8).astype(np.float32) for s in [(rows, n), (n,), (n,)]]
    _check(b.module([b.convert(z, dt) if dt != "f32" else z]), inputs, 2e-2 if dt != "f32" else 1e-5)


@pytest.mark.parametrize("shape,dim,dt", [((40, 30522 // 6), 1, "bf16"), ((64, 520), 1, "f32"), ((6, 4098), 1, "f32"), ((600, 66), 0, "bf16"), ((300, 64), 0, "bf16"),
                                          ((90, 70, 4), 0, "f32")])
def test_reductions_of_runs(shape, dim, dt):
    """Rows in pieces of 2, 4 and 8, columns in pieces of 2 and 4, with an operand along the columns (sums exact in any order)."""
    r = np.random.default_rng(shape[0])
    b = Builder()
    x, bias = b.arg(shape, dt), b.arg(shape[1:], dt)
    y = b.add(x, b.bcast(bias, shape, tuple(range(1, len(shape)))))
    y = b.convert(y, "f32") if dt != "f32" else y
    _check(b.module([b.reduce_sum(y, (dim,)), b.reduce_max(y, (dim,))]), [r.integers(-4, 5, s).astype(np.float32) for s in (shape, shape[1:])], 1e-6)


def test_many_wide_accumulators_fit_shared_memory():
    """Four sums in f64 over columns in runs of two, several runs a thread: fewer runs where their tiles would not fit."""
    import b200
    b = Builder()
    x = b.arg((600, 1026), "f64")
    sums = [b.reduce_sum(y, (0,)) for y in (x, b.mul(x, x), b.mul(x, b.mul(x, x)), b.neg(x))]
    plan, src = b200.compile_to_plan(b.module(sums), validate=True)
    import re
    for body in src.split('extern "C"')[1:]:
        tiles = re.findall(r"__shared__ double sm\d+\[(\d+)\]\[(\d+)\]", body)
        assert sum(int(r) * int(c) * 8 for r, c in tiles) <= 48 * 1024


@pytest.mark.parametrize("dt,parts,tanh,whole", [("f32", (96, 104), False, True), ("f32", (96, 104), True, False), ("f32", (128, 128), True, True), ("f32", (64, 64), True, False), ("bf16", (96, 104), True, False),
                                                 ("bf16", (384, 384), True, True), ("bf16", (256, 512), True, True), ("bf16", (96, 104), False, True), ("bf16", (100, 100), False, False), ("f32", (90, 110), False, False)])
def test_concatenations_of_runs(dt, parts, tanh, whole):
    """Two parts of a row: run by run where no run and few warps have the border inside, or where there is little to compute; each branch
    is then taken by a whole run. The values are those of the interpreter either way."""
    import re

    import b200
    rows = -(-151552 // sum(parts)) // 8 * 8 + 8
    r = np.random.default_rng(parts[0])
    b = Builder()
    xs = [b.arg((rows, n), dt) for n in parts]
    text = b.module([b.concatenate([b.tanh(x) if tanh else x for x in xs], 1)])
    src = b200.compile_to_plan(text, validate=True)[1]
    kernel = src[src.index('extern "C"'):]
    assert bool(re.search(r"reinterpret_cast<const uint4\*>\(in0 \+ l\d+\)", kernel)) == whole, kernel
    _check(text, [(np.round(r.standard_normal((rows, n)) * 8) / 8).astype(np.float32) for n in parts], 2e-2 if dt == "bf16" else 1e-6)
