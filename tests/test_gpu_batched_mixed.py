"""The shared-memory mixed batch kernel at the edges of its size classes:
backward error, independence of the batch around a system, and systems that
must reach the FP64 kernel."""
import numpy as np
import pytest

from conftest import EPS64

pytestmark = pytest.mark.gpu

EDGES = [1, 2, 7, 8, 9, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 163, 164, 165, 200, 231, 232, 233,
         234, 239, 240, 241, 255, 256]


def _systems(sizes, seed):
    rng = np.random.default_rng(seed)
    As, bs = [], []
    for n in sizes:
        As.append(np.asfortranarray(rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)[rng.permutation(n)]))
        bs.append(rng.standard_normal(n))
    return As, bs


def _solve(ctx, pkg, As, bs):
    bt = pkg.Batch(ctx, [a.shape[0] for a in As], "fp32")
    x = bt.solve(np.concatenate([a.ravel(order="F") for a in As]), np.concatenate(bs))
    it, info = bt.iterations(), bt.info.copy()
    bt.close()
    return np.split(x, np.cumsum([len(b) for b in bs])[:-1]), it, info


@pytest.mark.parametrize("copies", [1, 40])
def test_size_edges(ctx, pkg, oracle_mod, copies):
    """copies = 40: enough systems for one launch per size class."""
    sizes = EDGES * copies
    As, bs = _systems(sizes, 11)
    xs, it, info = _solve(ctx, pkg, As, bs)
    assert (info == 0).all() and (it >= 0).all()
    for a, b, x in zip(As[: 4 * len(EDGES)], bs, xs):
        assert oracle_mod.backward_error(a, x, b) <= 10 * len(b) * EPS64
    # the same systems alone give the same bits
    for i in (0, 5, 14, 19, 22, 23, len(EDGES) - 1):
        alone, _, _ = _solve(ctx, pkg, [As[i]], [bs[i]])
        assert np.array_equal(alone[0], xs[i])


@pytest.mark.parametrize("n", [5, 64, 130, 232, 240])
@pytest.mark.parametrize("kind", ["zero_column", "nan", "out_of_fp32_range"])
def test_fp64_resolve(ctx, pkg, oracle_mod, n, kind):
    """A zero pivot, a NaN or entries outside the FP32 range in one system:
    it goes to the FP64 kernel (the oracle's bits), its neighbours do not."""
    As, bs = _systems([n, n, n], n)
    if kind == "zero_column":
        As[1][:, n // 2] = 0.0
    elif kind == "nan":
        As[1][n // 3, 0] = np.nan
    else:
        As[1] *= 1e60
    xs, it, info = _solve(ctx, pkg, As, bs)
    assert it[0] >= 0 and it[1] == -1 and it[2] >= 0
    LU, ipiv, ref_info = oracle_mod.getrf(As[1])
    assert info[1] == ref_info
    if ref_info == 0:
        assert np.array_equal(xs[1], oracle_mod.getrs(LU, ipiv, bs[1]), equal_nan=True)
    for i in (0, 2):
        assert oracle_mod.backward_error(As[i], xs[i], bs[i]) <= 10 * n * EPS64
