"""The fused Gram-Schmidt launches of the GMRES refinement and the scaled FP32
correction at their edges: rows around a CTA's 256, every basis size up to the
restart length, one to eight columns, right-hand sides of extreme size."""
import numpy as np
import pytest

from conftest import EPS64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 255, 256, 257, 700])
@pytest.mark.parametrize("nrhs,restart,trans", [(1, 1, "N"), (3, 2, "T"), (8, 30, "N")])
def test_gmres_columns_alone_and_together(ctx, oracle_mod, n, nrhs, restart, trans):
    """Converged at the solver's own bound n eps, and each column the same bits
    as when it is solved alone."""
    rng = np.random.default_rng(17 * n + nrhs)
    A = rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)
    B = rng.standard_normal((n, nrhs)) * 10.0 ** rng.integers(-200, 200, nrhs)
    f = ctx.factor(n, n, "bf16")
    assert f.getrf(A) == 0
    X, st = f.solve_refined(B, trans, mode="gmres_ir", gmres_restart=restart, gmres_tol=1e-14)
    assert st["converged"] == 1, st
    # a basis norm is the root of a sum of squares: columns whose squares leave
    # the range take the FP64 fallback
    in_range = np.all((np.abs(B).max(axis=0) > 1e-140) & (np.abs(B).max(axis=0) < 1e140))
    assert not in_range or st["fell_back"] == 0, st
    Aop = A if trans == "N" else A.T
    for q in range(nrhs):
        # the bound plus the rounding of the check's own residual
        assert oracle_mod.backward_error(Aop, X[:, q:q + 1], B[:, q:q + 1]) <= 10 * n * EPS64
        xq, _ = f.solve_refined(B[:, q], trans, mode="gmres_ir", gmres_restart=restart, gmres_tol=1e-14)
        assert np.array_equal(xq, X[:, q])
    f.close()


@pytest.mark.parametrize("scale", [1e-310, 1e-300, 1.0, 1e300])
def test_correction_scales(ctx, oracle_mod, scale):
    """Right-hand sides whose power-of-two scale is subnormal or near the top
    of the range, beside a zero column."""
    n = 130
    rng = np.random.default_rng(3)
    A = rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)
    B = np.zeros((n, 3))
    B[:, 0] = rng.uniform(0.5, 1.0, n)
    B[:, 2] = rng.uniform(0.5, 1.0, n) * scale
    f = ctx.factor(n, n, "fp32")
    assert f.getrf(A) == 0
    for mode in ("ir", "gmres_ir"):
        X, st = f.solve_refined(B, mode=mode)
        # columns whose residual gets below the normal numbers (or, for GMRES,
        # whose squares leave the range) take the FP64 fallback
        assert st["fell_back"] == 0 or scale != 1.0, st
        assert np.all(X[:, 1] == 0.0) and np.all(np.isfinite(X))
        x1, _ = f.solve_refined(B[:, 0], mode=mode)
        assert np.array_equal(x1, X[:, 0])
        if scale > 1e-305:  # below, the residual itself is rounded to subnormals
            ref = np.linalg.solve(A, B[:, 2] / scale)
            # cond(A) is a few: n eps of backward error, both solvers
            assert np.abs(X[:, 2] / scale - ref).max() <= 100 * n * EPS64 * np.abs(ref).max()
    f.close()
