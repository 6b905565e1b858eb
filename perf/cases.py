"""The work whose speed is watched: whole programs through the client API, as a user's script runs them.

A case is a dict of plain values; `work` and `tolerance` read it, `prepare` makes what a program has in hand before the
call (inputs on the device, the compiled executable) and `run` makes one call. Programs come from b200.shlo.programs where
that module has them (the four model families of the benchmark configurations); the small ones are written out here.
Every input is drawn from the seed on the device.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "jax-mps_b200"))
import b200  # noqa: E402
from b200.shlo import programs  # noqa: E402
from b200.shlo.builder import Builder  # noqa: E402

SIZE = {"f32": 4, "bf16": 2, "f16": 2, "i32": 4, "ui8": 1}
TORCH = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16, "i32": torch.int32, "ui8": torch.uint8}
# decoder shapes: the benchmark's own (Gemma-2B-shaped) and two smaller ones of the same family
DECODERS = {"2b": dict(dim=2048, heads=8, head_dim=256, hidden=16384), "small": dict(dim=1024, heads=4, head_dim=256, hidden=4096),
            "tiny": dict(dim=512, heads=8, head_dim=64, hidden=2048)}


def listed():
    return [
        # a jitted scalar-sized function in a Python loop: nothing but the cost of a call
        {"name": "call_small", "kind": "call", "n": 48},
        # the same from host arrays to host arrays: a short image batch normalised before it is shown to a model
        {"name": "call_host", "kind": "host", "n": 80},
        # one SGD step of a two-layer classifier, f32, a batch and widths that fit no tile
        {"name": "mlp_f32_ragged", "kind": "mlp", "batch": 250, "in": 784, "hidden": 1000, "classes": 10, "dtype": "f32"},
        # the headline configuration of the benchmark: CIFAR ResNet18, batch 128, SGD with momentum
        {"name": "resnet18_b128", "kind": "resnet", "batch": 128},
        # the same step on a small shard, where its two hundred launches weigh most
        {"name": "resnet18_b20", "kind": "resnet", "batch": 20},
        # the recurrent configuration: two scans of 100 dependent iterations and Adam
        {"name": "lstm_t100_b64", "kind": "lstm", "steps": 100, "batch": 64, "in": 32, "hidden": 256},
        # the masked-language-model configuration, bf16
        {"name": "mlm_bf16_b32_s128", "kind": "mlm", "batch": 32, "seq": 128, "dim": 768, "heads": 12, "layers": 6, "vocab": 30522,
         "dtype": "bf16"},
        # the same family as a small f32 fine-tuning step on ragged sequences
        {"name": "mlm_f32_b6_s77", "kind": "mlm", "batch": 6, "seq": 77, "dim": 512, "heads": 8, "layers": 4, "vocab": 8003, "dtype": "f32"},
        # serving: the prompt in one pass ...
        {"name": "prefill_2b_p512", "kind": "prefill", "model": "2b", "layers": 18, "vocab": 256000, "prompt": 512, "dtype": "bf16"},
        # ... and greedy decoding behind it
        {"name": "decode_2b_n16", "kind": "decode", "model": "2b", "layers": 18, "vocab": 256000, "prompt": 512, "new": 16, "dtype": "bf16"},
        # sampling: the best 50 of a batch of vocabulary rows, and their probabilities
        {"name": "topk_b16_v30522", "kind": "rank", "batch": 16, "vocab": 30522, "k": 50},
        # ridge regression / Gaussian-process style solves: factor, then two triangular solves
        {"name": "solve_b8_n160", "kind": "solve", "batch": 8, "n": 160, "rhs": 12},
    ]


def _log(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    kind = rng.choice(["call", "host", "mlp", "resnet", "lstm", "mlm", "prefill", "decode", "rank", "solve"])
    if kind == "call":
        return {"kind": kind, "n": _log(rng, 1, 65536)}
    if kind == "host":
        return {"kind": kind, "n": _log(rng, 1, 1024)}
    if kind == "mlp":
        return {"kind": kind, "batch": _log(rng, 16, 4096), "in": _log(rng, 64, 2048), "hidden": _log(rng, 64, 4096),
                "classes": _log(rng, 2, 2000), "dtype": rng.choice(["f32", "bf16"])}
    if kind == "resnet":
        return {"kind": kind, "batch": _log(rng, 4, 128)}
    if kind == "lstm":
        return {"kind": kind, "steps": _log(rng, 10, 100), "batch": _log(rng, 4, 64), "in": _log(rng, 8, 64), "hidden": _log(rng, 32, 256)}
    if kind == "mlm":
        dim, heads = rng.choice([(256, 4), (512, 8), (768, 12)])
        return {"kind": kind, "batch": _log(rng, 2, 32), "seq": _log(rng, 16, 128), "dim": dim, "heads": heads, "layers": rng.randint(1, 6),
                "vocab": _log(rng, 1000, 30522), "dtype": rng.choice(["bf16", "f32"])}
    if kind in ("prefill", "decode"):
        case = {"kind": kind, "model": rng.choice(["2b", "small", "tiny"]), "layers": _log(rng, 2, 18), "vocab": _log(rng, 2000, 256000),
                "prompt": _log(rng, 16, 512)}
        if kind == "decode":
            case["new"] = _log(rng, 4, 16)
        case["dtype"] = rng.choice(["bf16", "f16"])
        return case
    if kind == "rank":
        vocab = _log(rng, 1000, 64000)
        # every position in order (k = 0: a full key / index sort, what nucleus sampling needs) or the best k
        return {"kind": kind, "batch": _log(rng, 1, 32), "vocab": vocab, "k": rng.choice([0, _log(rng, 1, 100)])}
    return {"kind": kind, "batch": _log(rng, 1, 32), "n": _log(rng, 8, 320), "rhs": _log(rng, 1, 64)}


# ---------------------------------------------------------------------------
# programs: (text, [(name, shape, dtype)] of the arguments, [(name, shape, dtype)] of the results)
# ---------------------------------------------------------------------------
def _call_program(c):
    n = c["n"]
    b = Builder()
    x, w, y = b.arg((n,), "f32"), b.arg((n,), "f32"), b.arg((n,), "f32")
    p = b.tanh(b.add(b.mul(x, w), b.full((n,), 0.5, "f32")))
    d = b.sub(p, y)
    text = b.module([p, b.mean(b.mul(d, d), (0,))], name="jit_f")
    return text, [(a, (n,), "f32") for a in "xwy"], [("p", (n,), "f32"), ("loss", (), "f32")]


def _host_program(c):
    shape = (c["n"], 32, 32, 3)
    b = Builder()
    x, mean, std = b.arg(shape, "ui8"), b.arg((3,), "f32"), b.arg((3,), "f32")
    v = b.div(b.convert(x, "f32"), b.full(shape, 255.0, "f32"))
    v = b.div(b.sub(v, b.bcast(mean, shape, (3,))), b.bcast(std, shape, (3,)))
    return b.module([v], name="jit_normalize"), [("images", shape, "ui8"), ("mean", (3,), "f32"), ("std", (3,), "f32")], [("v", shape, "f32")]


def _mlp_program(c):
    B, I, H, C, dt = c["batch"], c["in"], c["hidden"], c["classes"], c["dtype"]
    spec = [("w1", (I, H)), ("b1", (H,)), ("w2", (H, C)), ("b2", (C,))]
    b = Builder()
    P = [b.arg(s, dt) for _, s in spec]
    x, y = b.arg((B, I), dt), b.arg((B,), "i32")
    h = b.tanh(b.add(b.matmul(x, P[0]), b.bcast(P[1], (B, H), (1,))))
    z = b.add(b.matmul(h, P[2]), b.bcast(P[3], (B, C), (1,)))
    loss = programs.softmax_cross_entropy_int(b, b.convert(z, "f32") if dt != "f32" else z, y)
    grads = b.grad(loss, P)
    b.root.taping = False
    new = [b.sub(p, b.mul(g, b.full(p.shape, 0.1, dt))) for p, g in zip(P, grads)]
    args = [(n, s, dt) for n, s in spec] + [("x", (B, I), dt), ("y", (B,), "i32")]
    # the gradients come back beside the parameters, for the norm that a training loop logs
    res = [("loss", (), "f32")] + [("g." + n, s, dt) for n, s in spec] + [(n, s, dt) for n, s in spec]
    return b.module([loss, *grads, *new], name="jit_mlp_step"), args, res


def _rank_program(c):
    B, V, k = c["batch"], c["vocab"], c["k"]
    b = Builder()
    x = b.arg((B, V), "f32")
    if not k:
        keys, ids = b.sort([x, b.iota((B, V), "i32", 1)], 1, descending=True)
        return b.module([keys, ids], name="jit_argsort"), [("logits", (B, V), "f32")], [("keys", (B, V), "f32"), ("ids", (B, V), "i32")]
    vals, ids = b.top_k(x, k)
    e = b.exp(b.sub(vals, b.bcast(b.reduce_max(vals, (1,)), (B, k), (0,))))
    p = b.div(e, b.bcast(b.reduce_sum(e, (1,)), (B, k), (0,)))
    return b.module([p, ids], name="jit_top_k"), [("logits", (B, V), "f32")], [("p", (B, k), "f32"), ("ids", (B, k), "i32")]


def _solve_program(c):
    lead, n, k = (c["batch"],), c["n"], c["rhs"]
    b = Builder()
    a, r = b.arg(lead + (n, n), "f32"), b.arg(lead + (n, k), "f32")
    low = b.cholesky(a)
    x = b.triangular_solve(low, b.triangular_solve(low, r), transpose_a="TRANSPOSE")
    return b.module([low, x], name="jit_solve"), [("a", lead + (n, n), "f32"), ("r", lead + (n, k), "f32")], \
        [("l", lead + (n, n), "f32"), ("x", lead + (n, k), "f32")]


def _decoder_shape(c):
    return dict(DECODERS[c["model"]], layers=c["layers"], vocab=c["vocab"], dtype=c["dtype"])


def _program(c):
    kind = c["kind"]
    if kind in ("call", "host", "mlp", "rank", "solve"):
        return globals()[f"_{kind}_program"](c)
    if kind == "resnet":
        p = programs.resnet18_train_step(batch=c["batch"])
    elif kind == "lstm":
        p = programs.lstm_scan_train_step(steps=c["steps"], batch=c["batch"], in_dim=c["in"], hidden=c["hidden"])
    elif kind == "mlm":
        p = programs.distilbert_mlm_step(batch=c["batch"], seq=c["seq"], vocab=c["vocab"], dim=c["dim"], layers=c["layers"], heads=c["heads"],
                                         ffn=4 * c["dim"], dtype=c["dtype"])
    elif kind == "prefill":
        p = programs.gemma_prefill(prompt_len=c["prompt"], cache_len=c["prompt"] + 128, **_decoder_shape(c))
    else:
        p = programs.gemma_decode_loop(start=c["prompt"], new_tokens=c["new"], cache_len=c["prompt"] + 128, **_decoder_shape(c))
    return p.text, p.args, p.results


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _values(c, args, g):
    """One tensor per argument, on the device, drawn from the generator `g`."""
    def normal(shape, dtype, std=1.0):
        return torch.empty(shape, dtype=TORCH[dtype], device="cuda").normal_(0.0, std, generator=g)

    def integers(shape, hi, dtype="i32"):
        return torch.randint(0, hi, shape, generator=g, device="cuda", dtype=TORCH[dtype])

    def const(shape, dtype, v):
        return torch.full(shape, v, dtype=TORCH[dtype], device="cuda")

    kind = c["kind"]
    for name, shape, dtype in args:
        leaf = name.split(".")[-1]
        if kind == "solve" and name == "a":
            m = normal(shape, "f32")
            yield m @ m.transpose(1, 2) / shape[1] + 0.5 * torch.eye(shape[1], device="cuda")
        elif kind == "host":
            yield integers(shape, 256, "ui8") if name == "images" else torch.rand(shape, generator=g, device="cuda") * 0.2 + 0.3
        elif kind == "rank":
            yield normal(shape, dtype, 3.0)
        elif dtype == "i32":
            hi = {"resnet": 10, "mlp": c.get("classes")}.get(kind, c.get("vocab"))
            yield integers(shape, hi)
        elif kind == "mlm":
            if name == "mask":
                yield (torch.rand(shape, generator=g, device="cuda") < 0.15).float()
            elif name.endswith("ln.scale"):
                yield const(shape, dtype, 1.0)
            elif len(shape) == 1:
                yield normal(shape, dtype, 0.01)
            else:
                yield normal(shape, dtype, 0.02)
        elif kind in ("prefill", "decode"):
            if leaf.endswith("norm"):
                yield normal(shape, dtype, 0.05)
            elif leaf.endswith("_cache"):
                t = normal(shape, dtype)
                t[c["prompt"]:] = 0
                yield t
            elif leaf == "embed":
                yield normal(shape, dtype, shape[1] ** -0.5)
            else:                      # fan-in scale; what writes to the residual stream is scaled down by its depth
                depth = (2 * c["layers"]) ** -0.5 if leaf in ("wo", "w_down") else 1.0
                yield normal(shape, dtype, depth * shape[0] ** -0.5)
        elif kind == "resnet" and name.startswith("p."):
            yield normal(shape, dtype, math.sqrt(2.0 / math.prod(shape[:-1]))) if leaf == "kernel" else const(shape, dtype, 1.0 if leaf == "scale" else 0.0)
        elif kind == "resnet" and name.startswith("m."):
            yield normal(shape, dtype, 1e-3)
        elif kind == "lstm" and name[:2] in ("m.", "v."):
            yield const(shape, dtype, 0.0)
        elif kind in ("mlp", "lstm") and len(shape) == 2 and name not in ("x", "targets"):
            yield normal(shape, dtype, math.sqrt(1.0 / shape[0]))
        else:
            yield normal(shape, dtype, 0.1 if len(shape) == 1 and kind != "call" else 1.0)


_client = None
_executables = {}
_stage = None


def _put(t):
    """A device tensor as a buffer of the client, through pinned host memory."""
    global _stage
    size = t.numel() * t.element_size()
    if _stage is None or _stage.numel() < size:
        _stage = torch.empty(max(size, 64 << 20), dtype=torch.uint8, pin_memory=True)
    host = _stage[:size].view(t.dtype).view(t.shape)
    host.copy_(t)
    if t.dtype == torch.bfloat16:
        buf = _client.buffer_from_host(host.view(torch.int16).numpy().view(np.uint16), dtype="bf16")
    else:
        buf = _client.buffer_from_host(host.numpy())
    _client.synchronize()              # the staging memory is free again
    return buf


class Outputs(list):
    """The result buffers of one call. A user's program hands them to its next call as they are; here each becomes a tensor when
    it is read. All one-dimensional results of a type are read as one tensor: a training step has dozens, and some of them
    (the gradient of a key bias) are zero up to rounding, so that only their size against their siblings means anything."""

    def __init__(self, bufs, results):
        super().__init__(bufs)
        self.results = results

    def __iter__(self):
        _client.synchronize()
        flat = {}
        for buf, (_, shape, dtype) in zip(super().__iter__(), self.results):
            t = torch.as_tensor(_View(buf, shape, dtype), device="cuda")
            t = t.view(torch.bfloat16) if dtype == "bf16" else t
            if len(shape) == 1 and len(self.results) > 8:
                flat.setdefault(dtype, []).append(t)
            else:
                yield t
        for ts in flat.values():
            yield torch.cat(ts)


class _View:
    def __init__(self, buf, shape, dtype):
        self.buf = buf
        self.__cuda_array_interface__ = {"data": (buf.device_pointer(), False), "shape": tuple(shape), "version": 3,
                                         "typestr": {"f32": "<f4", "f16": "<f2", "bf16": "<i2", "i32": "<i4"}[dtype]}


class _State:
    pass


def prepare(case, seed):
    global _client
    if _client is None:
        _client = b200.Client(device_ordinal=0)
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _executables:
        text, args, results = _program(case)
        _executables[key] = (_client.compile(text), args, results)
    s = _State()
    s.exe, args, s.results = _executables[key]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    s.host = case["kind"] == "host"
    s.args = [t.cpu().numpy() if s.host else _put(t) for t in _values(case, args, g)]
    return s


def run(state):
    if state.host:
        return state.exe(*state.args)
    return Outputs(state.exe.execute(state.args), state.results)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    c, kind = case, case["kind"]
    if kind == "call":
        return {"bytes": 4.0 * (4 * c["n"] + 1), "flops": 8.0 * c["n"]}
    if kind == "host":
        return {"bytes": 3072.0 * c["n"] * 5 + 24, "flops": 4.0 * 3072 * c["n"]}
    if kind == "rank":
        out = c["k"] or c["vocab"]
        return {"bytes": 4.0 * c["batch"] * c["vocab"] + 8.0 * c["batch"] * out, "flops": 0.0}
    if kind == "solve":
        n, k, B = c["n"], c["rhs"], c["batch"]
        return {"bytes": 4.0 * B * (n * n * 1.5 + 2 * n * k), "flops": B * (n ** 3 / 3.0 + 2.0 * n * n * k)}
    if kind == "mlp":
        B, I, H, C, s = c["batch"], c["in"], c["hidden"], c["classes"], SIZE[c["dtype"]]
        params = I * H + H + H * C + C
        return {"bytes": s * (3.0 * params + B * I) + 4 * B + 4, "flops": 2.0 * B * (2 * I * H + 3 * H * C)}
    if kind == "resnet":
        params = sum(math.prod(s) for _, s in programs.resnet18_param_spec())
        # multiply-adds per image: 555 422 720 forward, three times that for a step less the first layer's input gradient
        return {"bytes": 16.0 * params + c["batch"] * (3072 + 1) * 4.0, "flops": 2.0 * c["batch"] * (3 * 555_422_720 - 1_769_472)}
    if kind == "lstm":
        T, B, I, H = c["steps"], c["batch"], c["in"], c["hidden"]
        params = (I + H) * 4 * H + 4 * H + 2 * H * 4 * H + 4 * H
        cell = ((I + H) + 2 * H) * 4 * H
        return {"bytes": 4.0 * (6 * params + T * B * I + B * H), "flops": 2.0 * T * B * (3 * cell - I * 4 * H)}
    if kind == "mlm":
        dim, S, L, V = c["dim"], c["seq"], c["layers"], c["vocab"]
        spec = programs.distilbert_param_spec(V, S, dim, L, 4 * dim)
        params = sum(math.prod(s) for _, s in spec)
        mac = L * (4 * dim * dim + 8 * dim * dim + 2 * S * dim) + dim * dim + dim * V
        return {"bytes": 2.0 * SIZE[c["dtype"]] * params, "flops": 6.0 * mac * c["batch"] * S}
    d = DECODERS[c["model"]]
    dim, heads, hd, hidden, L, V, P = d["dim"], d["heads"], d["head_dim"], d["hidden"], c["layers"], c["vocab"], c["prompt"]
    layer = dim * heads * hd * 2 + 2 * dim * hd + 3 * dim * hidden
    if kind == "prefill":
        # rows of the embedding that the prompt names, and the whole of it for the one row of logits
        nbytes = 2.0 * (L * layer + V * dim + 2 * L * (P + 128) * hd) + 4.0 * V
        flops = 2.0 * P * L * layer + 2.0 * V * dim + 2.0 * L * heads * P * (P + 1) * hd
        return {"bytes": nbytes, "flops": flops}
    n = c["new"]
    # the weights do not fit on the chip: every token reads them once more
    kv = sum(2 * L * (P + i + 1) * hd for i in range(n))
    return {"bytes": 2.0 * (n * (L * layer + V * dim) + kv), "flops": n * 2.0 * (L * layer + V * dim) + 4.0 * heads * kv / 2}


def tolerance(case):
    kind = case["kind"]
    if kind in ("call", "host"):
        return {"rel": 1e-6, "max": 1e-5}
    if kind == "rank":
        return {"rel": 1e-6, "max": 1e-5} if case["k"] else "exact"
    if kind == "solve":
        return {"rel": 1e-5, "max": 1e-3}
    if kind == "lstm":
        # the first Adam step moves a parameter by the sign of its gradient: one that is zero up to rounding may go either way
        return {"rel": 1e-4, "max": 0.1}
    if kind == "resnet":
        # a ReLU input within rounding of zero passes or drops a gradient: no two orders of 32-bit summation agree on all of
        # a million of them, and one in a million is a thousandth of the leaf's norm
        return {"rel": 1e-2, "max": 0.5}
    if kind in ("mlp", "mlm") and case["dtype"] == "f32":
        return {"rel": 1e-4, "max": 0.01}
    # 16-bit activations rounded at every layer; the generated ids are whole numbers and have to agree
    return {"rel": 2e-2, "max": 0.8}
