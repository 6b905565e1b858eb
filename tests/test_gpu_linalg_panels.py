"""Edges of the paneled factorization and of the warp-per-vector substitution: orders around the panel width of 32, the
narrower panels of long columns, f64, and the largest order whose unknowns stay in registers."""
import numpy as np
import pytest

from b200.shlo.builder import Builder
from oracle import interp
from util import run_gpu


def _spd(batch, n, dtype, seed=0):
    m = np.random.default_rng(seed).standard_normal((batch, n, n))
    return (m @ m.transpose(0, 2, 1) / n + 0.5 * np.eye(n)).astype(dtype)


@pytest.mark.gpu
@pytest.mark.parametrize("n,dtype", [(1, "f32"), (31, "f32"), (32, "f32"), (33, "f32"), (97, "f32"), (160, "f32"), (355, "f32"), (64, "f64"), (161, "f64")])
@pytest.mark.parametrize("lower", [True, False])
def test_cholesky_panels(client, n, dtype, lower):
    a = _spd(2, n, np.float64 if dtype == "f64" else np.float32)
    b = Builder()
    got, _ = run_gpu(client, b.module([b.cholesky(b.arg(a.shape, dtype), lower)]), [a])
    want = np.linalg.cholesky(a.astype(np.float64))
    want = want if lower else want.transpose(0, 2, 1)
    tol = 1e-12 if dtype == "f64" else 5e-6
    np.testing.assert_allclose(got[0], want, rtol=tol, atol=tol)


@pytest.mark.gpu
@pytest.mark.parametrize("n,k,dtype,left,lower,tr", [
    (1, 1, "f32", True, True, "NO_TRANSPOSE"), (31, 3, "f32", True, False, "NO_TRANSPOSE"), (32, 9, "f32", False, True, "TRANSPOSE"),
    (33, 4, "f32", True, True, "TRANSPOSE"), (160, 700, "f32", True, True, "NO_TRANSPOSE"), (359, 5, "f32", False, False, "NO_TRANSPOSE"),
    (1024, 2, "f32", True, True, "NO_TRANSPOSE"), (1025, 2, "f32", True, True, "NO_TRANSPOSE"), (97, 5, "f64", True, False, "TRANSPOSE"),
    (200, 3, "f64", False, True, "NO_TRANSPOSE")])
def test_triangular_solve_panels(client, n, k, dtype, left, lower, tr):
    np_t = np.float64 if dtype == "f64" else np.float32
    rng = np.random.default_rng(n)
    a = np.stack([np.linalg.cholesky(m) for m in _spd(2, n, np.float64, 1)]).astype(np_t)
    a = a if lower else np.ascontiguousarray(a.transpose(0, 2, 1))
    rhs = rng.standard_normal((2, n, k) if left else (2, k, n)).astype(np_t)
    b = Builder()
    text = b.module([b.triangular_solve(b.arg(a.shape, dtype), b.arg(rhs.shape, dtype), left_side=left, lower=lower, transpose_a=tr)])
    got, _ = run_gpu(client, text, [a, rhs])
    op = a.astype(np.float64) if tr == "NO_TRANSPOSE" else a.astype(np.float64).transpose(0, 2, 1)
    want = np.linalg.solve(op, rhs) if left else np.linalg.solve(op.transpose(0, 2, 1), rhs.transpose(0, 2, 1)).transpose(0, 2, 1)
    tol = 1e-11 if dtype == "f64" else 2e-5
    np.testing.assert_allclose(got[0], want, rtol=tol, atol=tol * np.abs(want).max())
