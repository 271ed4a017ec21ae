"""The residual product with each number of rows a CTA (64, 128 or 256, by the load
of the busiest SM): the refined solution's backward error, and one to eight
columns the same bits as alone."""
import numpy as np
import pytest

from conftest import EPS64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [121, 975, 1219, 1951, 3049])
def test_residual_row_choices(ctx, oracle_mod, pkg, n):
    A, B = pkg.workloads.shifted(n, 5, seed=n)
    f = ctx.factor(n, n, "fp32")
    f.getrf(A)
    X, st = f.solve_refined(B)
    assert st["fell_back"] == 0, st
    assert oracle_mod.backward_error(A, X, B) <= 10 * n * EPS64
    x, _ = f.solve_refined(B[:, 4])
    assert np.array_equal(x, X[:, 4])
    f.close()
