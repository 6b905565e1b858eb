"""Chains of row kernels: rows of a few elements, units between two stages that read the chain but not by rows and what is filled with them, reshapes on both
sides of a softmax, rows of one block of 1024 threads. The generated kernels run on the CPU and are held to the interpreter."""
import shutil

import numpy as np
import pytest

if shutil.which("g++") is None:
    pytest.skip("needs g++ to build the generated kernels for the host", allow_module_level=True)

import b200
from b200.shlo import programs
from b200.shlo.builder import Builder
from cuda_emu import run_plan_on_cpu
from oracle import interp


def _check(text, inputs, tol):
    for g, w in zip(run_plan_on_cpu(text, inputs), interp.run_text(text, inputs), strict=True):
        np.testing.assert_allclose(np.asarray(g, np.float64), np.asarray(w, np.float64), rtol=tol, atol=tol)


@pytest.mark.parametrize("rows,classes", [(250, 10), (33, 2), (7, 3), (1, 31), (1025, 17)])
def test_cross_entropy_over_a_few_classes(rows, classes):
    """The mean over the rows stands between the stages; the gradient behind it is a stage again."""
    r = np.random.default_rng(rows)
    b = Builder()
    z, y = b.arg((rows, classes), "f32"), b.arg((rows,), "i32")
    loss = programs.softmax_cross_entropy_int(b, z, y)
    text = b.module([loss, *b.grad(loss, [z])])
    plan = b200.compile_to_plan(text)[0]
    assert plan.count(" row{") == 1 and plan.count("exponential") == 1, plan
    _check(text, [r.standard_normal((rows, classes)).astype(np.float32), r.integers(0, classes, rows).astype(np.int32)], 1e-5)


@pytest.mark.parametrize("dt,tol", [("f32", 1e-5), ("bf16", 2e-2)])
def test_softmax_between_reshapes(dt, tol):
    r = np.random.default_rng(1)
    b = Builder()
    x, m = b.arg((6 * 5, 64), dt), b.arg((5, 64), "f32")
    s = b.reshape(b.convert(x, "f32") if dt != "f32" else x, (6, 5, 64))
    s = b.add(b.mul(s, b.full(s.shape, 0.5, "f32")), b.bcast(m, s.shape, (1, 2)))
    e = b.exp(b.sub(s, b.bcast(b.reduce_max(s, (2,)), s.shape, (0, 1))))
    p = b.div(e, b.bcast(b.reduce_sum(e, (2,)), s.shape, (0, 1)))
    q = b.reshape(p, (30, 64))
    q = b.convert(q, dt) if dt != "f32" else q
    text = b.module([q])
    plan = b200.compile_to_plan(text)[0]
    assert plan.count("kernel ") == 1, plan
    _check(text, [(np.round(r.standard_normal((30, 64)) * 8) / 8).astype(np.float32), r.standard_normal((5, 64)).astype(np.float32)], tol)


def test_a_block_of_1024_threads():
    r = np.random.default_rng(2)
    b = Builder()
    x = b.arg((2, 8194), "f32")
    e = b.exp(b.sub(x, b.bcast(b.reduce_max(x, (1,)), x.shape, (0,))))
    text = b.module([b.div(e, b.bcast(b.reduce_sum(e, (1,)), x.shape, (0,)))])
    assert "block=1024x1" in b200.compile_to_plan(text)[0]
    _check(text, [r.standard_normal((2, 8194)).astype(np.float32)], 1e-6)


@pytest.mark.parametrize("rows,cols", [(64, 64), (7, 33)])
def test_a_broadcast_of_what_stands_behind_the_chain(rows, cols):
    """The sum over all rows is made behind the chain of rows, and so is the tensor filled with it."""
    r = np.random.default_rng(rows)
    b = Builder()
    t = b.arg((rows, cols), "f32")
    s = b.reduce_sum(t, (1,))
    q = b.reduce_sum(b.mul(s, s), (0,))
    filled = b.bcast(q, (rows, cols), ())
    text = b.module([b.sub(t, b.bcast(s, t.shape, (0,))), filled])
    plan = b200.compile_to_plan(text)[0]
    assert plan.count(" row{") == 1, plan
    _check(text, [r.standard_normal((rows, cols)).astype(np.float32)], 1e-5)
