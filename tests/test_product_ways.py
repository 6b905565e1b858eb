"""Which kernels an fp32 product goes to where its operands have no rows of 16 bytes: on both sides of the lines at which the FMA pipe and
the table-driven kernels were measured to take the same time. Plans only."""
import pytest

import b200
from b200.shlo.builder import Builder


@pytest.mark.parametrize("form,M,K,N,fma", [("nn", 200, 24323, 16, False), ("nn", 64, 7034, 64, False), ("tt", 8, 6495, 16, False), ("nn", 64, 62062, 32, False),
                                            ("nt", 256, 7938, 16, True), ("nn", 64, 3742, 32, True), ("tt", 30, 2289, 64, True), ("nn", 250, 1000, 10, True)])
def test_long_sums_of_single_floats(form, M, K, N, fma):
    b = Builder()
    x, y = b.arg((K, M) if form[0] == "t" else (M, K), "f32"), b.arg((N, K) if form[1] == "t" else (K, N), "f32")
    plan = b200.compile_to_plan(b.module([b.dot_general(x, y, ((0,) if form[0] == "t" else (1,), (1,) if form[1] == "t" else (0,)))]))[0]
    assert (" fma " in plan) == fma, plan
