"""The environment variables that the planner reads: all of them are part of a cached plan's key, with their values, and documented."""
import re
from pathlib import Path

import numpy as np
import pytest

from b200.shlo.builder import Builder

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "jax-mps_b200" / "csrc"


def _read(*names):
    text = "".join((CSRC / n).read_text() for n in names)
    return set(re.findall(r'getenv\("(B200_\w+)"\)', text))


def test_the_key_names_all_of_them():
    source = (CSRC / "compiler.cc").read_text()
    names = source[source.index("std::string planning_switches()"):]
    assert _read("compiler.cc", "loops.cc", "codegen.cc", "parser.cc") == set(re.findall(r'"(B200_\w+)"', names[:names.index("return s;")]))


def test_all_variables_are_documented():
    documented = set(re.findall(r"B200_\w+", (ROOT / "INTEGRATION.md").read_text()))
    assert _read(*(f.name for f in CSRC.glob("*.c*"))) <= documented


@pytest.mark.gpu
@pytest.mark.parametrize("name,values", [("B200_NO_HELD_ROWS", [None, "1"]), ("B200_ROW_WARP_MAX", [None, "64", "128"]), ("B200_NO_WIDE_ROWS", [None, "1"])])
def test_each_setting_has_its_plan(client, monkeypatch, name, values):
    b = Builder()
    x = b.arg((2048, 96), "f32")
    e = b.exp(b.sub(x, b.bcast(b.reduce_max(x, (1,)), x.shape, (0,))))
    text = b.module([b.div(e, b.bcast(b.reduce_sum(e, (1,)), x.shape, (0,)))], name="jit_switches")
    a = np.random.default_rng(0).standard_normal((2048, 96)).astype(np.float32)
    want = np.exp(a.astype(np.float64) - a.max(1, keepdims=True))
    kept = []
    for v in values:
        monkeypatch.delenv(name, raising=False) if v is None else monkeypatch.setenv(name, v)
        kept.append(client.compile(text))
        np.testing.assert_allclose(kept[-1](a)[0], want / want.sum(1, keepdims=True), rtol=1e-5, atol=1e-7)
    # 96 elements a row: a warp each up to 128, a block beyond 64
    assert len({exe.fingerprint for exe in kept}) == 2
