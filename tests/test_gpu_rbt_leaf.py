"""The 128-column no-pivot leaf of the butterfly-transformed factors at its
edges: ragged last leaves, sub-block boundaries, rows below the leaf around a
CTA's 32, and the trailing solves through the inverse the leaf leaves behind."""
import numpy as np
import pytest

from conftest import EPS64
from test_gpu_mixed import _rbt_matrices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "fp16"])
@pytest.mark.parametrize("n", [4, 31, 33, 97, 127, 128, 129, 159, 161, 255, 256, 385, 641])
def test_leaf_factors(ctx, oracle_mod, pkg, prec, n):
    A, B = pkg.workloads.shifted(n, 2, seed=900 + n)
    f = ctx.factor(n, n, prec)
    f.set_pivoting("rbt")
    assert f.getrf(A) == 0
    U_, V_ = _rbt_matrices(n)
    Ar = U_.T @ A @ V_
    F = f.factors()
    L, U = np.tril(F, -1) + np.eye(n), np.triu(F)
    # the standard bound n u |L||U|, u that of the update's operands, times 8
    # for the block inverses (their condition is a few: A is diagonally
    # dominant) and 8 u for the transform, itself a sum of 16 terms
    u = 2.0 ** -24 if prec == "fp32" else 2.0 ** -11
    bound = 8 * n * u * (np.abs(L) @ np.abs(U)).max() + 8 * 2.0 ** -24 * np.abs(Ar).max()
    assert np.abs(Ar - L @ U).max() <= bound
    for trans in ("N", "T"):
        X, st = f.solve_refined(B, trans)
        assert st["fell_back"] == 0, st
        assert oracle_mod.backward_error(A if trans == "N" else A.T, X, B) <= 10 * n * EPS64
    f.close()


@pytest.mark.parametrize("n", [40, 130, 300])
def test_leaf_zero_pivot(ctx, n):
    """A zero matrix: the first pivot is exactly zero."""
    f = ctx.factor(n, n, "fp32")
    f.set_pivoting("rbt")
    f.getrf(np.eye(n))
    assert np.array_equal(f.ipiv(), np.arange(1, n + 1))
    f.close()
    g = ctx.factor(n, n, "bf16")
    g.set_pivoting("rbt")
    A = np.zeros((n, n))
    try:
        info = g.getrf(A)
    except Exception:
        info = 1  # the FP64 fallback found it singular
    assert info == 1
    g.close()
