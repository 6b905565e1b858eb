"""The factorization that keeps its matrix in registers (f32, 33 to 208 rows) and the substitution by blocks of eight unknowns:
orders around the tiles of four, the panels of sixteen and the blocks, one and several tiles a thread, both triangles, matrices
that are not positive definite (NaN from the first bad pivot on) or out of the range of the quick root. The generated kernels run
on the CPU and are held to float64 (n rounded operations in a row: n times 2^-23 of the result's scale) and to the interpreter."""
import shutil

import numpy as np
import pytest

if shutil.which("g++") is None:
    pytest.skip("needs g++ to build the generated kernels for the host", allow_module_level=True)

from b200.shlo.builder import Builder
from cuda_emu import run_plan_on_cpu


def _spd(n, seed=0):
    m = np.random.default_rng(seed).standard_normal((2, n, n))
    return (m @ m.transpose(0, 2, 1) / n + 0.5 * np.eye(n)).astype(np.float32)


@pytest.mark.parametrize("n,scale", [(33, 1.0), (48, 1.0), (50, 1e-32), (67, 1e32), (141, 1.0), (166, 1.0), (208, 1.0)])
@pytest.mark.parametrize("lower", [True, False])
def test_resident_cholesky(n, scale, lower):
    a = (_spd(n).astype(np.float64) * scale).astype(np.float32)
    b = Builder()
    got = run_plan_on_cpu(b.module([b.cholesky(b.arg(a.shape, "f32"), lower)]), [a])[0].astype(np.float64)
    want = np.linalg.cholesky(a.astype(np.float64))
    want = want if lower else want.transpose(0, 2, 1)
    np.testing.assert_allclose(got, want, rtol=0, atol=n * 2.0 ** -23 * np.abs(want).max())


@pytest.mark.parametrize("n", [33, 50, 67, 141])
def test_rows_past_the_matrix_are_zero(n):
    """... in both panels that the tile warps read, of shared memory that is full of NaNs to begin with."""
    check = """  if (u == 0)
    for (int h = 0; h < 2; ++h)
      for (int k = 0; k < NB; ++k)
        for (int r = N; r < NP; ++r)
          if (((const T*)final4[h])[k * NP + r] != (T)0) o[0] = __uint_as_float(0x7FC00000u);
"""
    def edit(src):
        at = src.index("#undef AT", src.index("final4"))
        return src[:at] + check + src[at:]
    b = Builder()
    a = _spd(n)
    got = run_plan_on_cpu(b.module([b.cholesky(b.arg(a.shape, "f32"))]), [a], edit)[0]
    np.testing.assert_allclose(got, np.linalg.cholesky(a.astype(np.float64)), rtol=0, atol=n * 2.0 ** -23 * 4)


def test_resident_cholesky_of_an_indefinite_matrix():
    n = 52
    a = _spd(n)
    a[1, 37, 37] = -1.0
    a += np.triu(np.full((n, n), np.nan, np.float32), 1)                              # only the lower triangle is read
    b = Builder()
    got = run_plan_on_cpu(b.module([b.cholesky(b.arg(a.shape, "f32"))]), [a])[0]
    np.testing.assert_allclose(got[0], np.linalg.cholesky(np.nan_to_num(a[0]).astype(np.float64)), rtol=0, atol=1e-5)
    np.testing.assert_allclose(got[1][:37, :37], np.linalg.cholesky(np.nan_to_num(a[1][:37, :37]).astype(np.float64)), rtol=0, atol=1e-5)
    assert np.isnan(got[1][37:, 37]).all() and np.isnan(got[1][51, 51]) and (np.triu(got[1], 1) == 0).all()


@pytest.mark.parametrize("n,k", [(7, 1), (8, 3), (9, 2), (31, 1), (40, 9), (65, 3)])
@pytest.mark.parametrize("left,lower,tr,unit", [(True, True, "NO_TRANSPOSE", False), (True, True, "TRANSPOSE", False), (False, False, "NO_TRANSPOSE", False), (True, False, "NO_TRANSPOSE", True)])
def test_substitution_by_blocks(n, k, left, lower, tr, unit):
    r = np.random.default_rng(n)
    low = np.linalg.cholesky(_spd(n, 1).astype(np.float64)).astype(np.float32)
    a = low if lower else np.ascontiguousarray(low.transpose(0, 2, 1))
    if unit:
        a = (a * (1 - np.eye(n)) * 0.3 + np.eye(n) * 7).astype(np.float32)           # the diagonal is not read
    rhs = r.standard_normal((2, n, k) if left else (2, k, n)).astype(np.float32)
    b = Builder()
    got = run_plan_on_cpu(b.module([b.triangular_solve(b.arg(a.shape, "f32"), b.arg(rhs.shape, "f32"), left_side=left, lower=lower, unit_diagonal=unit, transpose_a=tr)]),
                          [a, rhs])[0]
    op = a.astype(np.float64)
    if unit:
        op = op * (1 - np.eye(n)) + np.eye(n)
    op = op.transpose(0, 2, 1) if tr == "TRANSPOSE" else op
    want = np.linalg.solve(op, rhs) if left else np.linalg.solve(op.transpose(0, 2, 1), rhs.transpose(0, 2, 1)).transpose(0, 2, 1)
    np.testing.assert_allclose(got, want, rtol=0, atol=4 * n * 2.0 ** -23 * np.abs(want).max())
