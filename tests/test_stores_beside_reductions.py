"""A column sum whose first pass also stores a pointwise result over the same elements, in front of a chain of row kernels: the
result is made once, in the rows that the 16-bit product behind it reads (padded where their length is no multiple of eight), and
so is what the second pass makes of the sums. On the GPU held to float64: tanh and the product are rounded to 8 bits once each
(2e-2 of the result's scale), the sums of 4096 values are fp32."""
import re

import numpy as np
import pytest

import b200
from b200.shlo.builder import Builder, f32_to_bf16_bits
from util import run_gpu


def program(rows, cols, lanes=128):
    b = Builder()
    g, t, w = b.arg((rows, cols), "bf16"), b.arg((rows, lanes), "f32"), b.arg((cols, 64), "bf16")
    m = b.reduce_max(t, (1,))
    sums = b.reduce_sum(b.convert(g, "f32"), (0,))
    y, scaled = b.tanh(g), b.sin(sums)
    e = b.exp(b.sub(t, b.bcast(m, t.shape, (0,))))
    z = b.div(e, b.bcast(b.reduce_sum(e, (1,)), t.shape, (0,)))
    return b.module([sums, scaled, z, b.matmul(y, w)], name=f"jit_beside_{rows}_{cols}")


@pytest.mark.parametrize("cols", [1024, 1026, 1030, 2050])
def test_made_once(cols):
    plan = b200.compile_to_plan(program(4096, cols))[0]
    assert plan.count("tanh") == 1 and plan.count("sine") == 1 and "repack16" not in plan, plan
    first = next(line for line in plan.splitlines() if "tanh" in line)
    assert "reduce_" in first and plan.index(first) < plan.index("row{"), plan


@pytest.mark.gpu
@pytest.mark.parametrize("cols", [1024, 1026, 1028, 1030, 1284, 2050])
def test_values(client, cols):
    r = np.random.default_rng(cols)
    def bf16(*shape): return (f32_to_bf16_bits(r.standard_normal(shape).astype(np.float32)).astype(np.uint32) << 16).view(np.float32)
    g, t, w = bf16(4096, cols), r.standard_normal((4096, 128)).astype(np.float32), bf16(cols, 64)
    (sums, scaled, z, o), _ = run_gpu(client, program(4096, cols), [g, t, w], ["bf16", None, "bf16"])
    want = g.astype(np.float64).sum(0)
    np.testing.assert_allclose(sums, want, rtol=1e-5, atol=1e-5 * np.abs(want).max())
    np.testing.assert_allclose(scaled, np.sin(sums.astype(np.float64)), rtol=1e-5, atol=1e-5)
    e = np.exp(t.astype(np.float64) - t.max(1, keepdims=True))
    np.testing.assert_allclose(z, e / e.sum(1, keepdims=True), rtol=1e-5, atol=1e-7)
    want = np.tanh(g.astype(np.float64)) @ w.astype(np.float64)
    np.testing.assert_allclose(np.asarray(o, np.float64), want, rtol=2e-2, atol=2e-2 * np.abs(want).max())


def _kernel(src, name):
    body = src[src.index(f" {name}("):]
    return body[:body.index("\n}\n")]


@pytest.mark.parametrize("rows,wide", [(2_080_000, False), (2_090_000, True)])
def test_padded_rows_past_32_bits(rows, wide):
    """2 090 000 rows of 1026 elements are below 2^31, 1032 apart they are not."""
    assert rows * 1026 < 2**31 - 65536 and (rows * 1032 >= 2**31) == wide
    b = Builder()
    g, w = b.arg((rows, 1026), "bf16"), b.arg((1026, 64), "bf16")
    plan, src = b200.compile_to_plan(b.module([b.reduce_sum(b.convert(g, "f32"), (0,)), b.matmul(b.tanh(g), w)]), validate=True)
    assert "partial+fusion{tanh}" in plan, plan
    assert ("(i64)x0 * 1032" if wide else "(int)x0 * 1032") in _kernel(src, "reduce_0")


@pytest.mark.parametrize("kind", ["rows", "columns", "chain", "chain of two reads"])
def test_slices_of_a_tensor_past_32_bits(kind):
    """10 000 of 3 000 000 rows of 1024: the reduction is small, where it reads is not."""
    b = Builder()
    x = b.arg((3_000_000, 1024), "bf16")
    y = b.convert(b.slice(x, [2_990_000, 0], [3_000_000, 1024]), "f32")
    s = b.reduce_sum(y, (0 if kind == "columns" else 1,))
    outs = [b.rsqrt(s), b.tanh(s)] if kind == "chain" else [s]
    if kind == "chain of two reads":
        outs = [b.mul(b.bcast(s, y.shape, (0,)), b.convert(b.slice(x, [1_990_000, 0], [2_000_000, 1024]), "f32"))]
    plan, src = b200.compile_to_plan(b.module(outs), validate=True)
    assert ("row{" in plan) == kind.startswith("chain"), plan
    readers = [k for k in src.split('extern "C"')[1:] if "const u16* __restrict__ in" in k]
    assert readers and all("const i64 " in k for k in readers)


@pytest.mark.parametrize("n,wide", [(2**31 - 3_000_000, False), (2**31 - 2_000_000, True), (2**31 - 100_000, True)])
def test_the_step_past_the_end_of_a_row(n, wide):
    """A row shared by a thousand blocks: the index that ends a thread's loop lies up to two million elements past the row."""
    b = Builder()
    plan, src = b200.compile_to_plan(b.module([b.reduce_sum(b.arg((n,), "f32"), (0,))]), validate=True)
    splits = int(plan.split("grid=1x")[1].split()[0])
    assert splits > 1000, plan
    loop = next(line for line in _kernel(src, "reduce_0").splitlines() if "gridDim.y" in line and "for (" in line)
    step = 256 * (4 if "* 4;" in loop else 1) * splits
    assert (n + step >= 2**31) <= wide
    assert loop.strip().startswith("for (i64 " if wide else "for (int "), loop


@pytest.mark.parametrize("cols,groups", [(1022, 1), (1024, 2), (1026, 1), (1028, 2), (30522, 1), (30524, 2)])
def test_one_run_of_columns_a_thread(cols, groups):
    """Two runs a thread only where the pass stores a tensor as well and a run is 16 bytes of f32; no branch between the loads of a
    thread."""
    for stores in (False, True):
        b = Builder()
        g = b.arg((8192, cols), "f32")
        plan, src = b200.compile_to_plan(b.module([b.reduce_sum(g, (0,))] + ([b.tanh(g)] if stores else [])), validate=True)
        kernel = _kernel(src, "reduce_0")
        assert plan.splitlines()[1].endswith("args=[2,3,0]" if stores else "args=[2,0]"), plan
        assert f"float acc0[{(4 if cols % 4 == 0 else 2) * (groups if stores else 1)}]" in kernel
        rows = kernel[kernel.index("for (int r = "):]
        assert "break" not in rows[:rows.index("\n  }\n")]


def test_two_runs_of_wide_accumulators_fit_shared_memory():
    b = Builder()
    x = b.arg((4096, 1028), "f32")
    y = b.convert(x, "f64")
    plan, src = b200.compile_to_plan(b.module([b.reduce_sum(v, (0,)) for v in (y, b.mul(y, y), b.mul(y, b.mul(y, y)), b.neg(y))] + [b.tanh(x)]), validate=True)
    assert "+fusion{tanh}" in plan, plan
    tiles = re.findall(r"__shared__ double sm\d+\[(\d+)\]\[(\d+)\]", _kernel(src, "reduce_0"))
    assert len(tiles) == 4 and sum(int(r) * int(c) * 8 for r, c in tiles) <= 48 * 1024


@pytest.mark.parametrize("rows,cols,one_pass", [(65536, 64, True), (131072, 66, False), (100000, 100, False), (65536, 128, True), (32768, 130, True), (49152, 86, True), (45000, 94, True),
                                                (32768, 132, False), (16384, 514, True)])
def test_one_pass_where_rows_fill_its_threads(rows, cols, one_pass):
    b = Builder()
    x = b.arg((rows, cols), "f32")
    plan = b200.compile_to_plan(b.module([b.reduce_sum(x, (0,)), b.tanh(x)]))[0]
    assert ("+fusion{tanh}" in plan) == one_pass, plan
