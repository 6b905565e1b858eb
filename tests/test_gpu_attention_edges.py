"""Decode attention at the ends of its range: whole chunks, just over a whole number of chunks, 32 and 33 chunks,
the smallest and largest rows, eight query rows (whose sums are halved across the lanes) and seven."""
import numpy as np
import pytest

from b200.shlo.programs import decode_attention as attention_program
from oracle import interp
from test_attention import _inputs
from util import run_gpu


@pytest.mark.gpu
@pytest.mark.parametrize("G,M,T,D,N", [(2, 8, 32, 256, 256), (None, 7, 33, 256, 8), (3, 8, 65, 8, 256), (None, 8, 1024, 16, 24), (2, 7, 1025, 64, 40)])
def test_ends_of_the_range(client, G, M, T, D, N):
    text = attention_program(G, M, T, D, N, "bf16", True, True)
    args = _inputs(G, M, T, D, N) + [np.array(T - 1, np.int32)]
    assert "attention_" in client.compile(text).plan_text()
    got, _ = run_gpu(client, text, args, dtypes=["bf16"] * 3 + ["i32"])
    want = interp.run_text(text, [np.asarray(a) for a in args])
    np.testing.assert_allclose(np.asarray(got[0], np.float64), np.asarray(want[0], np.float64), rtol=2e-2, atol=2e-2)
