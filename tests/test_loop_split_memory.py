"""What a counted loop costs in memory when its sums leave it: 512 MB at most, whatever the operands of a sum are made of, and
nothing where one of them is the same in all iterations; and which products leave: those that take less time as one. Plans only: no
step of these sizes is run."""
import re

import pytest

import b200
from b200.shlo import programs
from b200.shlo.builder import Builder


def sums(T, R, I, N, form):
    """dw += a^T g[t], db += the rows of g[t], over t; `a` is a tensor that does not change ("same"), a function of one ("made"),
    the slice x[t] ("rows"), x[T-1-t] ("reversed"), or carried from iteration to iteration ("carried")."""
    b = Builder()
    x, g = b.arg((R, I) if form in ("same", "made", "carried") else (T, R, I), "f32"), b.arg((T, R, N), "f32")

    def at(s, v, t): return s.reshape(s.dynamic_slice(v, [t, s.const(0, "i32"), s.const(0, "i32")], (1, *v.shape[1:])), v.shape[1:])

    def body(s, k, dw, db, h):
        gt = at(s, g, s.sub(s.const(T - 1, "i32"), k) if form == "reversed" else k)
        a = {"same": lambda: x, "made": lambda: s.tanh(x), "rows": lambda: at(s, x, k), "reversed": lambda: at(s, x, s.sub(s.const(T - 1, "i32"), k)),
             "carried": lambda: h}[form]()
        return [s.add(k, s.const(1, "i32")), s.add(dw, s.dot_general(a, gt, ((0,), (0,)))), s.add(db, s.reduce_sum(gt, (0,))), s.tanh(h)]
    start = x if form == "carried" else b.full((1, 1), 0.5, "f32")
    _, dw, db, h = b.while_([b.const(0, "i32"), b.full((I, N), 0.0, "f32"), b.full((N,), 0.0, "f32"), start], lambda s, k, *r: s.compare(k, s.const(T, "i32"), "LT"), body)
    return b.module([dw, db, h], name=f"jit_sums_{T}_{R}_{I}_{N}_{form}")


def _arena(plan):
    return int(re.search(r"arena0 (\d+) bytes", plan).group(1))


# whether the product over all iterations stands behind the loop
CASES = [("same", 400, 4096, 1024, 64, False), ("same", 12000, 4096, 1024, 2, False), ("same", 16, 64, 64, 64, False), ("made", 16, 64, 64, 64, True),
         ("made", 400, 4096, 1024, 64, False), ("rows", 1000, 64, 1024, 16, True), ("rows", 1001, 64, 1024, 16, True), ("rows", 2001, 64, 1024, 16, False),
         ("rows", 65536, 2, 64, 64, True), ("reversed", 1000, 64, 1024, 16, True), ("reversed", 1800, 64, 1024, 16, True), ("reversed", 1900, 64, 1024, 16, False),
         ("carried", 100, 64, 256, 64, True), ("carried", 900, 64, 1024, 16, True), ("carried", 1100, 64, 1024, 16, False)]


@pytest.mark.parametrize("form,T,R,I,N,taken", CASES)
def test_scratch_of_sums_behind_a_loop(monkeypatch, form, T, R, I, N, taken):
    text = sums(T, R, I, N, form)
    split = b200.compile_to_plan(text)[0]
    monkeypatch.setenv("B200_NO_LOOP_SPLIT", "1")
    whole = b200.compile_to_plan(text)[0]
    assert _arena(split) - _arena(whole) <= 512 << 20, split
    assert any(line.startswith("  igemm") for line in split.splitlines()) == taken, split
    assert taken or _arena(split) <= _arena(whole), (split, whole)


def recurrence(T, R, I, N):
    """h = tanh([x[t], y[T-1-t]] w + h): the product is made in front of the loop from a concatenation of a slice and a reversed one."""
    b = Builder()
    x, y, w, h0 = b.arg((T, R, I), "f32"), b.arg((T, R, I), "f32"), b.arg((2 * I, N), "f32"), b.arg((R, N), "f32")

    def at(s, v, t): return s.reshape(s.dynamic_slice(v, [t, s.const(0, "i32"), s.const(0, "i32")], (1, *v.shape[1:])), v.shape[1:])

    def body(s, k, h):
        a = s.concatenate([at(s, x, k), at(s, y, s.sub(s.const(T - 1, "i32"), k))], 1)
        return [s.add(k, s.const(1, "i32")), s.tanh(s.add(s.matmul(a, w), h))]
    return b.module([b.while_([b.const(0, "i32"), h0], lambda s, k, *r: s.compare(k, s.const(T, "i32"), "LT"), body)[1]], name=f"jit_front_{T}_{R}_{I}_{N}")


@pytest.mark.parametrize("T,R,I,N,taken", [(100, 64, 32, 1024, True), (900, 64, 256, 1024, True), (1300, 64, 256, 1024, False), (2500, 64, 256, 16, True),
                                           (6000, 64, 256, 16, False)])
def test_scratch_of_a_product_in_front_of_a_loop(monkeypatch, T, R, I, N, taken):
    text = recurrence(T, R, I, N)
    split = b200.compile_to_plan(text)[0]
    monkeypatch.setenv("B200_NO_LOOP_SPLIT", "1")
    whole = b200.compile_to_plan(text)[0]
    assert any(line.startswith("  igemm") for line in split.splitlines()) == taken, split
    assert _arena(split) - _arena(whole) <= (512 << 20 if taken else 0), split


# batch and hidden size of a two-layer recurrent training step, products made in front of the reverse loop, sums of products behind it
STEPS = [(4, 32, 2, 2), (16, 256, 2, 2), (64, 256, 2, 2), (64, 512, 2, 2), (16, 1024, 2, 2), (256, 256, 2, 0), (256, 512, 1, 0), (256, 1024, 0, 0), (512, 512, 0, 0)]


@pytest.mark.parametrize("batch,hidden,front,behind", STEPS)
def test_products_leave_where_that_is_quicker(monkeypatch, batch, hidden, front, behind):
    text = programs.lstm_scan_train_step(steps=50, batch=batch, in_dim=8, hidden=hidden).text
    split = b200.compile_to_plan(text)[0]
    monkeypatch.setenv("B200_NO_LOOP_SPLIT", "1")
    whole = b200.compile_to_plan(text)[0]
    assert _arena(split) - _arena(whole) <= 512 << 20
    outside = [line for line in split.splitlines() if line.startswith("  igemm")]
    assert all(" fma " in line for line in outside), split
    assert sum(f"M={50 * batch} " in line for line in outside) == front, split
    assert len({line.split("N=")[1].split()[0] + line.split("M=")[1].split()[0] for line in outside if f"M={50 * batch} " not in line}) == behind, split


def test_a_product_of_a_transposed_operand_stays():
    """x[t]^T w: all iterations' of them are not one matrix, and would not run where an iteration's do."""
    T, R, I, N = 20, 32, 64, 48
    b = Builder()
    x, w, h0 = b.arg((T, R, I), "f32"), b.arg((R, N), "f32"), b.arg((I, N), "f32")

    def body(s, k, h):
        xt = s.reshape(s.dynamic_slice(x, [k, s.const(0, "i32"), s.const(0, "i32")], (1, R, I)), (R, I))
        return [s.add(k, s.const(1, "i32")), s.tanh(s.add(s.dot_general(xt, w, ((0,), (0,))), h))]
    plan = b200.compile_to_plan(b.module([b.while_([b.const(0, "i32"), h0], lambda s, k, *r: s.compare(k, s.const(T, "i32"), "LT"), body)[1]]))[0]
    assert [line for line in plan.splitlines() if "igemm" in line and " fma " in line and line.startswith("    ")], plan
    assert not any(line.startswith("  igemm") for line in plan.splitlines()), plan


@pytest.mark.parametrize("rows,again", [(1, True), (100, True), (148, True), (149, False), (256, False)])
def test_small_values_of_a_body_are_made_again(monkeypatch, rows, again):
    """Two carried tensors made of one exponential: each of their kernels makes it for itself while a block on each of 148 SMs covers
    it (151 552 elements), beyond that it is made once. The switch of the split is not the one of this."""
    b = Builder()
    x, y = b.arg((rows, 1024), "f32"), b.arg((1024, rows), "f32")

    def body(s, k, h, t):
        e = s.exp(s.tanh(h))
        return [s.add(k, s.const(1, "i32")), s.mul(e, s.full(e.shape, 0.5, "f32")), s.add(s.transpose(e, (1, 0)), t)]
    text = b.module(b.while_([b.const(0, "i32"), x, y], lambda s, k, *r: s.compare(k, s.const(10, "i32"), "LT"), body)[1:])
    for name in (None, "B200_NO_LOOP_SPLIT", "B200_NO_LOOP_RECOMPUTE"):
        with monkeypatch.context() as m:
            if name:
                m.setenv(name, "1")
            plan = b200.compile_to_plan(text)[0]
        assert plan.count("exponential") == (2 if again and name != "B200_NO_LOOP_RECOMPUTE" else 1), (name, plan)
