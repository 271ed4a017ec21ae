"""The exact getrs sweeps where they can go wrong: several right-hand sides
(one CTA each), ragged blocks, quotients outside the range of the FMA division,
zero dividends and NaN; and the fast transposed sweeps."""
import numpy as np
import pytest

from conftest import EPS64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 64, 97, 128, 193, 321])
@pytest.mark.parametrize("nrhs", [1, 2, 5, 8, 9])
@pytest.mark.parametrize("trans", ["N", "T"])
def test_exact_sweeps_bit_exact(ctx, oracle_mod, n, nrhs, trans):
    rng = np.random.default_rng(n * 13 + nrhs)
    A = rng.standard_normal((n, n))
    B = rng.standard_normal((n, nrhs))
    f = ctx.factor(n, n)
    f.getrf(A)
    LU, ipiv, _ = oracle_mod.getrf(A)
    assert np.array_equal(f.getrs(B, trans), oracle_mod.getrs(LU, ipiv, B, trans))
    f.close()


@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("kind", ["zeros", "unit", "tiny_b", "huge_b", "wide_diagonal", "nan"])
def test_exact_sweeps_division_range(ctx, oracle_mod, trans, kind):
    """Where the quotient or the reciprocal leaves the safe range (or is zero)
    the sweeps fall back to the IEEE division, four columns at a time."""
    n = 150
    rng = np.random.default_rng(5)
    A = rng.standard_normal((n, n)) + 10 * np.eye(n)
    B = rng.standard_normal((n, 3))
    if kind == "zeros":
        B[:] = 0.0
        B[70, 1] = -0.0
    elif kind == "unit":
        B[:] = 0.0
        B[[0, 64, 149], [0, 1, 2]] = 1.0
    elif kind == "tiny_b":
        B *= 1e-305
    elif kind == "huge_b":
        B *= 1e300
    elif kind == "wide_diagonal":
        A = np.diag(10.0 ** rng.integers(-300, 300, n).astype(float))  # its own U
    else:
        B[40, 0] = np.nan
    f = ctx.factor(n, n)
    f.getrf(A)
    LU, ipiv, _ = oracle_mod.getrf(A)
    X, Xo = f.getrs(B, trans), oracle_mod.getrs(LU, ipiv, B, trans)
    assert np.array_equal(X, Xo, equal_nan=True)
    assert np.array_equal(np.signbit(X[~np.isnan(Xo)]), np.signbit(Xo[~np.isnan(Xo)]))
    f.close()


@pytest.mark.parametrize("n,nrhs", [(64, 2), (65, 1), (700, 5), (1025, 9)])
def test_fast_transposed_sweeps(ctx, oracle_mod, n, nrhs):
    """Backward error of op(A) = A^T within the bound the fast mode is held to
    (10 n eps), one right-hand side per CTA or several."""
    rng = np.random.default_rng(n)
    A = np.asfortranarray(rng.standard_normal((n, n)))
    B = rng.standard_normal((n, nrhs))
    f = ctx.factor(n, n)
    f.getrf(A)
    f.set_solve("fast")
    X = f.getrs(B, "T")
    assert oracle_mod.backward_error(A.T, X, B) <= 10 * n * EPS64
    f.close()


@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("bits", [0xFFFFFFFFFFFFFFFF, 0x7FFFFFFFFFFFFFFF, 0xFFF4FFF4FFF4FFF4, 0xFFFCFFF4FFF4FFF4])
@pytest.mark.parametrize("where", ["b", "diagonal", "above", "below", "last"])
def test_exact_sweeps_nan_payloads(ctx, oracle_mod, trans, bits, where):
    """NaN whose payload FP64 arithmetic carries along, the all-ones pattern of
    a buffer filled with 0xFF among them: NaN comes out where the oracle has
    it, and no sweep waits for a value that is there."""
    n = 150
    rng = np.random.default_rng(8)
    A = np.asfortranarray(rng.standard_normal((n, n)) + 10 * np.eye(n))
    B = np.asfortranarray(rng.standard_normal((n, 3)))
    nan = np.array([bits], dtype=np.uint64)
    if where == "b":
        B.view(np.uint64)[40, 1] = nan[0]
    else:
        A.view(np.uint64)[{"diagonal": (70, 70), "above": (10, 120), "below": (120, 10), "last": (n - 1, n - 1)}[where]] = nan[0]
    f = ctx.factor(n, n)
    f.getrf(A)
    LU, ipiv, _ = oracle_mod.getrf(A)
    assert np.array_equal(f.factors(), LU, equal_nan=True)
    X, Xo = f.getrs(B, trans), oracle_mod.getrs(LU, ipiv, B, trans)
    assert np.isnan(Xo).any()
    assert np.array_equal(X, Xo, equal_nan=True)
    f.close()
