"""A program that comes back is replayed as a graph whose branches run side by side: the replays must give the bits of the
first, step by step execution, whichever buffers they get, and a program is recorded once."""
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
    return b.module([b.add(left, b.broadcast_in_dim(m, (64, 96), (0,))), rows, *keys, vals, pos, b.reduce_sum(right, (0, 1)), w]), \
        [((64, 96), "f32"), ((96, 96), "f32"), ((200,), "i32")]


def _program(name):
    if name == "everything":
        return _everything()
    p = {"resnet": lambda: programs.resnet18_train_step(batch=4, image=16, width=8),
         "lstm": lambda: programs.lstm_scan_train_step(steps=41, batch=5, in_dim=8, hidden=24),
         "decode": lambda: programs.gemma_decode_loop(vocab=160, dim=64, layers=2, heads=2, head_dim=32, hidden=128, start=9, new_tokens=11, cache_len=24, dtype="bf16"),
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


def _arrays(args, rng):
    for shape, dtype in args:
        yield rng.integers(0, 10, shape).astype(np.int32) if dtype == "i32" else (rng.standard_normal(shape) * 0.3).astype(np.float32)


def _buffers(client, args, arrays):
    return [client.buffer_from_host(a) if d == "i32" else client.buffer_from_host(a, dtype=d) for (_, d), a in zip(args, arrays)]


@pytest.fixture(scope="module")
def by_steps():
    """A client that records nothing."""
    import os
    import b200
    names = ["B200_NO_PLAN_GRAPHS", "B200_NO_LOOP_GRAPHS"]
    for n in names:
        os.environ[n] = "1"
    try:
        c = b200.Client()
    finally:
        for n in names:
            del os.environ[n]
    yield c
    c.synchronize()


def _loops(name):
    return {"lstm": 2, "decode": 1}.get(name, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["everything", "resnet", "lstm", "mlm", "decode"])
def test_new_buffers_need_no_new_recording(client, by_steps, name):
    """Every call has buffers of its own, and all of them and all results stay alive, so that no address comes back."""
    text, args = _program(name)
    exe, plain = client.compile(text), by_steps.compile(text)
    rng = np.random.default_rng(1)
    before = exe.recordings
    kept = []
    for k in range(6):
        arrays = list(_arrays(args, rng))
        kept.append((exe.execute(_buffers(client, args, arrays)), plain.execute(_buffers(by_steps, args, arrays)), arrays))
    for got, want, _ in kept:
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g.to_numpy(), w.to_numpy())
    graphs = max(1, _loops(name))
    assert exe.recordings - before <= graphs
    assert exe.relocations >= 4 * graphs
    assert plain.recordings == 0


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["resnet", "lstm"])
def test_a_training_loop_is_recorded_once(client, by_steps, name):
    """State fed back, a fresh batch in every step: the bits of the loop that is run step by step, and one recording."""
    p = {"resnet": lambda: programs.resnet18_train_step(batch=4, image=16, width=8),
         "lstm": lambda: programs.lstm_scan_train_step(steps=43, batch=5, in_dim=8, hidden=24)}[name]()
    args = [(s, d) for _, s, d in p.args]
    names, state = [a[0] for a in p.args], [r[0] for r in p.results]
    first = programs.resnet18_inputs(p) if name == "resnet" else programs.lstm_inputs(p)
    fresh = [i for i, n in enumerate(names) if n not in state]
    losses = []
    for c in (client, by_steps):
        exe = c.compile(p.text)
        before = exe.recordings
        rng = np.random.default_rng(2)
        bufs = _buffers(c, args, first)
        run = []
        for _ in range(12):
            for i in fresh:
                a = np.array(first[i])
                bufs[i] = c.buffer_from_host(rng.permutation(a.reshape(-1)).reshape(a.shape))
            outs = exe.execute(bufs)
            for n, o in zip(state, outs):
                if n in names:
                    bufs[names.index(n)] = o
            run.append(outs[0])
        losses.append([o.to_numpy() for o in run] + [o.to_numpy() for o in outs])
        assert exe.recordings - before <= (max(1, _loops(name)) if c is client else 0)
    for g, w in zip(*losses):
        np.testing.assert_array_equal(g, w)


@pytest.mark.gpu
def test_arguments_may_be_one_buffer(client, by_steps):
    """A recording made while two arguments were one buffer serves calls in which they are two, and the other way about."""
    b = Builder()
    x, y = b.arg((96, 96), "f32"), b.arg((96, 96), "f32")
    h = b.matmul(b.tanh(b.matmul(x, y)), x)
    text = b.module([b.matmul(b.sub(h, y), y), b.reduce_sum(b.mul(h, x), (0,)), x, y, b.transpose(b.add(x, h), (1, 0))])
    exe, plain = client.compile(text), by_steps.compile(text)
    rng = np.random.default_rng(3)
    for k, one in enumerate([True, True, False, False, True, False]):
        a, c = (rng.standard_normal((96, 96)).astype(np.float32) for _ in range(2))
        got, want = [], []
        for to, cl, e in ((got, client, exe), (want, by_steps, plain)):
            u = cl.buffer_from_host(a)
            v = u if one else cl.buffer_from_host(c)
            to += [o.to_numpy() for o in e.execute([u, v])]
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g, w)
    assert exe.recordings == 1 and exe.relocations >= 2
