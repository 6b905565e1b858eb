"""Constants and index tables are on the device before the first kernel that reads them, also when a program is executed as soon as it is
compiled and behind large transfers."""
import re
from pathlib import Path

import numpy as np
import pytest

from b200.shlo.builder import Builder

RUNTIME = Path(__file__).resolve().parent.parent / "jax-mps_b200" / "csrc" / "runtime.cc"


def test_nothing_goes_to_the_device_on_the_default_stream():
    """The client's streams do not wait for the default stream, and what is sent on it may arrive after the call."""
    source = re.sub(r"//[^\n]*", "", RUNTIME.read_text())
    assert not re.findall(r"cudaMemset\(|cudaMemcpy\([^;]*cudaMemcpyHostToDevice", source)
    assert "cudaStreamNonBlocking" in source


@pytest.mark.gpu
def test_products_by_tables_right_behind_their_compilation(client, monkeypatch):
    """Operands of 3 to 40 MB on their way while the tables (0.1 to 1.5 MB) of one product after the other are sent, in the memory of
    the one before."""
    monkeypatch.setenv("B200_NO_GEMM32", "1")
    monkeypatch.setenv("B200_NO_TILE32", "1")
    r = np.random.default_rng(0)
    for k, (M, K, N) in enumerate([(64, 40001, 16), (8, 6495, 16), (200, 24323, 16), (30, 55187, 32), (64, 7034, 64), (400, 10001, 60)] * 4):
        b = Builder()
        x, y = b.arg((M, K), "f32"), b.arg((K, N), "f32")
        text = b.module([b.matmul(x, y)], name=f"jit_tables_{k}")
        a, c = r.integers(-3, 4, (M, K)).astype(np.float32), r.integers(-3, 4, (K, N)).astype(np.float32)
        bufs = [client.buffer_from_host(v) for v in (a, c)]
        out = client.compile(text).execute(bufs)[0].to_numpy()
        np.testing.assert_allclose(out, a.astype(np.float64) @ c.astype(np.float64), rtol=1e-5, atol=1e-3)
