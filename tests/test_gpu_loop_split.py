"""Counted loops whose products and sums leave the loop: a recurrence with stacked carries and its reverse pass, over trip counts
that do and do not divide into whole sums, counters that do not start at zero, rows walked both ways; and loops that look alike
but have to stay as they are. Held to the oracle and to the loop as it stands (f32; the sums over iterations are of the same
length as in the loop or shorter, so the bound is that of a product: 1e-5 of the result's scale)."""
import numpy as np
import pytest

from b200.shlo.builder import Builder
from oracle import interp


def recurrence(T, B, I, H, first=0, form="plain"):
    """h' = tanh(x[t] W + h U); backwards in time g -> (g * (1 - z^2)) U^T with z = tanh(h[t] V) recomputed from the stacked h,
    and the sums over time of h[t]^T z-gradients, of the gradients' rows, and of something that only looks like such a sum."""
    b = Builder()
    xs, w, u, v, g0 = b.arg((T, B, I), "f32"), b.arg((I, H), "f32"), b.arg((H, H), "f32"), b.arg((H, H), "f32"), b.arg((B, H), "f32")
    limit = b.arg((), "i32") if form == "dynamic" else None

    def c(s, n): return s.const(n, "i32")
    def at(s, stack, t): return s.reshape(s.dynamic_slice(stack, [t, c(s, 0), c(s, 0)], (1, *stack.shape[1:])), stack.shape[1:])
    def cond(s, k, *r): return s.compare(k, limit if limit is not None else c(s, first + T), "LT")

    def fwd(s, k, h, hs):
        t = s.sub(k, c(s, first)) if first else k
        hs2 = s.dynamic_update_slice(hs, s.reshape(h, (1, B, H)), [t, c(s, 0), c(s, 0)])
        return [s.add(k, c(s, 1)), s.tanh(s.add(s.matmul(at(s, xs, t), w), s.matmul(h, u))), hs2]
    zero = b.full((B, H), 0.0, "f32")
    start = b.const(first, "i32")
    _, h_last, hs = b.while_([start, zero, b.full((T, B, H), 0.0, "f32")], cond, fwd)

    def bwd(s, k, g, dv, db, other):
        t = s.sub(c(s, first + T - 1 + (2 if form == "clamped" else 0)), k)
        h = at(s, hs, t)
        z = s.tanh(s.matmul(h, v))
        dz = s.mul(g, s.sub(s.full((B, H), 1.0, "f32"), s.mul(z, z)))
        term = s.dot_general(h, dz, ((0,), (0,)))
        if form == "read":                                # the accumulator is read by the iteration: it has to stay
            dz = s.add(dz, s.mul(s.bcast(db, (B, H), (1,)), s.full((B, H), 1e-3, "f32")))
        g2 = s.dot_general(dz, u, ((1,), (1,)))
        return [s.add(k, c(s, 2 if form == "strided" else 1)), g2, s.add(dv, term), s.add(s.reduce_sum(dz, (0,)), db), s.mul(s.add(other, term if form == "shared" else s.bcast(s.reduce_sum(g2, (0,)), (H, H), (1,))), s.full((H, H), 0.5, "f32"))]
    _, g, dv, db, other = b.while_([start, g0, b.full((H, H), 0.25, "f32"), b.full((H,), -1.0, "f32"), b.full((H, H), 0.0, "f32")], cond, bwd)
    r = np.random.default_rng(T + B + H)
    args = [r.standard_normal((T, B, I)), r.standard_normal((I, H)) / I ** 0.5, r.standard_normal((H, H)) * 0.5 / H ** 0.5, r.standard_normal((H, H)) / H ** 0.5,
            r.standard_normal((B, H))]
    args = [a.astype(np.float32) for a in args] + ([np.array(first + T, np.int32)] if limit is not None else [])
    return b.module([h_last, g, dv, db, other], name=f"jit_rec_{T}_{B}_{I}_{H}_{first + 10}_{form}"), args


CASES = [(8, 3, 5, 7, 0, "plain"), (13, 64, 32, 40, 0, "plain"), (17, 100, 8, 33, 3, "plain"), (100, 6, 4, 16, 0, "plain"), (9, 600, 4, 20, -2, "plain"), (16, 32, 8, 64, 1, "plain"),
         (7, 4, 4, 8, 0, "plain"), (12, 5, 4, 8, 0, "shared"), (12, 5, 4, 8, 0, "dynamic"), (12, 5, 4, 8, 0, "clamped"), (12, 5, 4, 8, 0, "read"), (12, 5, 4, 8, 0, "strided")]


@pytest.mark.gpu
@pytest.mark.parametrize("T,B,I,H,first,form", CASES)
def test_split_loops(client, monkeypatch, T, B, I, H, first, form):
    text, args = recurrence(T, B, I, H, first, form)
    exe = client.compile(text)
    plan = exe.plan_text()
    assert (f"M={T * B} N={H} K={H}" in plan) == (T >= 8 and form in ("plain", "read", "shared")), plan
    got = exe(*args)
    again = exe(*args)
    monkeypatch.setenv("B200_NO_LOOP_SPLIT", "1")
    whole = client.compile(text)(*args)
    for a, a2, w, o in zip(got, again, whole, interp.run_text(text, args, wide=True), strict=True):
        np.testing.assert_array_equal(a, a2)
        scale = np.abs(o).max()
        np.testing.assert_allclose(a, o, rtol=1e-5, atol=1e-5 * scale)
        np.testing.assert_allclose(a, w, rtol=1e-5, atol=1e-5 * scale)
