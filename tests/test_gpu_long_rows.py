"""Cross entropy over a large vocabulary in 16 bits, forward and backward: rows that one block of 1024 threads holds in registers,
the gradient of the logits stored by the pass that sums its columns (in rows padded for the products that read it where the
vocabulary is not a multiple of eight), and, from 2^25 logits on, exponentials made again instead of stored. Held to float64; the
gradient is rounded to 8 bits once and the logits once before it, so 2e-2 of a result's scale bounds both."""
import numpy as np
import pytest

from b200.shlo import programs
from b200.shlo.builder import Builder
from util import run_gpu


def _bf16(x):
    u = np.asarray(x, np.float32).view(np.uint32).astype(np.uint64)
    return (((u + 0x7FFF + ((u >> 16) & 1)) >> 16) << 16).astype(np.uint32).view(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,vocab", [(160, 30522), (300, 16390), (200, 30520), (1150, 30522), (149, 65534)])
def test_cross_entropy_over_a_vocabulary(client, rows, vocab):
    r = np.random.default_rng(rows)
    h, w = _bf16(r.standard_normal((rows, 64)) * 0.5), _bf16(r.standard_normal((vocab, 64)) * 0.3)
    bias, label = r.standard_normal(vocab).astype(np.float32) * 0.1, r.integers(0, vocab, rows).astype(np.int32)
    b = Builder()
    hv, wv, bv, lv = b.arg(h.shape, "bf16"), b.arg(w.shape, "bf16"), b.arg(bias.shape, "f32"), b.arg(label.shape, "i32")
    z = b.add(b.convert(b.dot_general(hv, wv, ((1,), (1,))), "f32"), b.bcast(bv, (rows, vocab), (1,)))
    loss = programs.softmax_cross_entropy_int(b, z, lv)
    text = b.module([loss, *b.grad(loss, [hv, wv, bv])], name=f"jit_ce_{rows}_{vocab}")
    plan = client.compile(text).plan_text()
    assert "block=1024x1 row{" in plan and "repack16" not in plan, plan
    stored = next(line for line in plan.splitlines() if "row{" in line)
    assert (stored.count("exponential") > 1) == (rows * vocab >= 1 << 25), plan
    got, _ = run_gpu(client, text, [h, w, bias, label], ["bf16", "bf16", None, None])
    z64 = _bf16(h.astype(np.float64) @ w.astype(np.float64).T).astype(np.float64) + bias
    z64 -= z64.max(1, keepdims=True)
    p = np.exp(z64)
    s = p.sum(1, keepdims=True)
    np.testing.assert_allclose(got[0], np.mean(np.log(s[:, 0]) - z64[np.arange(rows), label]), rtol=1e-3)
    p /= s
    p[np.arange(rows), label] -= 1.0
    p /= rows
    for g, want in zip(got[1:], (p @ w, p.T @ h, p.sum(0))):
        np.testing.assert_allclose(np.asarray(g, np.float64), want, rtol=2e-2, atol=2e-2 * np.abs(want).max())
