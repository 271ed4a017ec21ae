"""The fast sweeps' clusters at their edges: block-row counts below, at and past
a cluster of eight, ragged last block rows (whose tiles take partial 16-byte
copies), odd right-hand-side counts."""
import numpy as np
import pytest

from conftest import EPS64

pytestmark = pytest.mark.gpu

SIZES = [1, 64, 67, 130, 255, 449, 512, 513, 577, 1090]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("trans", ["N", "T"])
def test_fp64_fast_sweeps(ctx, oracle_mod, n, trans):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)
    B = rng.standard_normal((n, 3))
    f = ctx.factor(n, n)
    f.set_solve("fast")
    f.getrf(A)
    X = f.getrs(B, trans)
    assert oracle_mod.backward_error(A if trans == "N" else A.T, X, B) <= 10 * max(n, 4) * EPS64
    assert np.array_equal(f.getrs(B[:, 1], trans), X[:, 1])
    f.close()


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("nrhs", [1, 2, 3, 8])
def test_fp32_fast_sweeps(ctx, oracle_mod, n, nrhs):
    """Through refinement, which takes more than a few steps (or falls back) if a
    correction solve is wrong; each column the same bits as alone."""
    rng = np.random.default_rng(n + nrhs)
    A = rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)
    B = rng.standard_normal((n, nrhs))
    f = ctx.factor(n, n, "fp32")
    f.getrf(A)
    for trans in ("N", "T"):
        X, st = f.solve_refined(B, trans)
        # each step gains the FP32 solve's relative error, 1e-4 or better here:
        # three steps reach n eps, a fourth is for rounding
        assert st["fell_back"] == 0 and st["iterations"] <= 4, st
        assert oracle_mod.backward_error(A if trans == "N" else A.T, X, B) <= 10 * max(n, 4) * EPS64
        x, _ = f.solve_refined(B[:, nrhs - 1], trans)
        assert np.array_equal(x, X[:, nrhs - 1])
    f.close()
