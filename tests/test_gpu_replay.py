"""Programs that come back with the same addresses are replayed as graphs whose branches run side by side: the replays must
give the bits of the first, step by step execution, also when the inputs changed in between."""
import numpy as np
import pytest

from b200.shlo import programs
from b200.shlo.builder import Builder


def _everything():
    """Independent branches, products, a sort, a scatter and values that many steps read."""
    b = Builder()
    x, w, i = b.arg((64, 96), "f32"), b.arg((96, 96), "f32"), b.arg((200,), "i32")
    h = b.matmul(x, w)
    left, right = b.matmul(b.tanh(h), w), b.dot_general(h, x, ((1,), (1,)))
    rows = b.scatter_rows(b.full((300, 96), 1.0, "f32"), i, b.broadcast_in_dim(b.reduce_sum(left, (0,)), (200, 96), (1,)), "add")
    keys = b.sort([b.reshape(right, (4096,)), b.iota((4096,), "i32", 0)], 0)
    m = b.reduce_max(left, (1,))
    vals, pos = b.top_k(b.reshape(left, (1, 64 * 96)), 5)
    return b.module([b.add(left, b.broadcast_in_dim(m, (64, 96), (0,))), rows, *keys, vals, pos, b.reduce_sum(right, (0, 1))]), \
        [((64, 96), "f32"), ((96, 96), "f32"), ((200,), "i32")]


def _program(name):
    if name == "everything":
        return _everything()
    p = {"resnet": lambda: programs.resnet18_train_step(batch=4, image=16, width=8),
         "lstm": lambda: programs.lstm_scan_train_step(steps=41, batch=5, in_dim=8, hidden=24),
         "mlm": lambda: programs.distilbert_mlm_step(batch=2, seq=16, vocab=200, dim=64, layers=2, heads=4, ffn=128, dtype="bf16")}[name]()
    return p.text, [(s, d) for _, s, d in p.args]


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["everything", "resnet", "lstm", "mlm"])
def test_replays_repeat_the_first_execution(client, name):
    text, args = _program(name)
    exe = client.compile(text)
    rng = np.random.default_rng(0)

    def inputs():
        return [client.buffer_from_host(rng.integers(0, 10, s).astype(np.int32)) if d == "i32" else
                client.buffer_from_host((rng.standard_normal(s) * 0.3).astype(np.float32), dtype=d) for s, d in args]
    sets = [inputs(), inputs()]
    want = [[o.to_numpy() for o in exe.execute(s)] for s in sets]
    for k in range(8):
        got = [o.to_numpy() for o in exe.execute(sets[k % 2])]
        for g, w in zip(got, want[k % 2]):
            np.testing.assert_array_equal(g, w)
    client.synchronize()
