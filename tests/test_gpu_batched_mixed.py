"""The shared-memory mixed batch kernel at the edges of its size classes:
backward error, independence of the batch around a system, and systems that
must reach the FP64 kernel."""
import ctypes
import subprocess

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


@pytest.mark.parametrize("n,count", [(80, 1500), (150, 900), (200, 500), (240, 500)])
def test_singular_systems_leave_the_others_alone(ctx, pkg, n, count):
    """More systems than CTAs, every third one with a zero FP32 pivot (all zero,
    a zero column, entries below the FP32 range): the systems that follow in
    the same CTA are refined and have the bits they have without them."""
    rng = np.random.default_rng(n)
    As = rng.standard_normal((count, n, n)) + 2 * np.sqrt(n) * np.eye(n)
    bs = rng.standard_normal((count, n))
    bad = np.arange(count) % 3 == 1
    kind = np.arange(count) // 3 % 3
    As[bad & (kind == 0)] = 0.0
    As[bad & (kind == 1), n // 2, :] = 0.0  # stored by columns: a zero column
    As[bad & (kind == 2)] *= 1e-60

    def solve(sel):
        bt = pkg.Batch(ctx, [n] * int(sel.sum()), "fp32")
        x = bt.solve(As[sel].ravel(), bs[sel].ravel()).reshape(-1, n)
        it, info = bt.iterations(), bt.info.copy()
        bt.close()
        return x, it, info

    x, it, info = solve(np.ones(count, bool))
    xg, itg, infog = solve(~bad)
    assert (itg >= 0).all() and (infog == 0).all()
    assert np.array_equal(it[~bad], itg)
    assert np.array_equal(x[~bad], xg)
    assert (it[bad] == -1).all()
    assert (info[bad & (kind == 0)] == 1).all()
    assert (info[bad & (kind == 1)] == n // 2 + 1).all()
    tiny = bad & (kind == 2)
    assert (info[tiny] == 0).all()
    r = np.einsum("sji,sj->si", As[tiny], x[tiny]) - bs[tiny]  # row i of A is As[:, i]
    scale = np.abs(As[tiny]).sum(1).max(1) * np.abs(x[tiny]).max(1) + np.abs(bs[tiny]).max(1)
    assert (np.abs(r).max(1) <= 10 * n * EPS64 * scale).all()


def test_size_class_residency(ctx, pkg):
    """A class whose CTAs have 256 threads or fewer is one of which an SM holds
    several; a CTA alone on an SM has 512."""
    pkg.Batch(ctx, [8], "fp32").close()  # the kernels are set up with the first batch
    per_sm = ctx.lib._ZN4gblu23batch_mixed_ctas_per_smEiPi
    threads = ctypes.c_int()
    for n in range(1, 257):
        ctas = per_sm(n, ctypes.byref(threads))
        assert ctas >= (2 if threads.value <= 256 else 1), (n, threads.value, ctas)


@pytest.mark.parametrize("n", [157, 159, 160, 161])
def test_pair_class_edge(ctx, pkg, oracle_mod, n):
    """The last size of which two fit an SM and the first that has one alone,
    in one batch: the bits each system has by itself."""
    sizes = [n, 161, n, 160] * 90
    As, bs = _systems(sizes, n)
    xs, it, info = _solve(ctx, pkg, As, bs)
    assert (info == 0).all() and (it >= 0).all()
    for i in range(4):
        assert oracle_mod.backward_error(As[i], xs[i], bs[i]) <= 10 * sizes[i] * EPS64
        alone, _, _ = _solve(ctx, pkg, [As[i]], [bs[i]])
        assert np.array_equal(alone[0], xs[i])


RESIDUAL_C = """
#include <math.h>
void residual(long n, const double *a, const double *x, const double *b, double *r) {
  for (long i = 0; i < n; ++i) {
    double s = b[i];
    for (long j = 0; j < n; ++j) s = fma(-a[i + j * n], x[j], s);
    r[i] = s;
  }
}
"""


@pytest.fixture(scope="module")
def residual(tmp_path_factory):
    d = tmp_path_factory.mktemp("residual")
    (d / "r.c").write_text(RESIDUAL_C)
    subprocess.run(["gcc", "-O2", "-shared", "-fPIC", "-o", str(d / "r.so"), str(d / "r.c"), "-lm"], check=True)
    f = ctypes.CDLL(str(d / "r.so")).residual
    f.argtypes = [ctypes.c_long] + 4 * [ctypes.c_void_p]
    f.restype = None

    def call(a, x, b):
        r = np.empty_like(b)
        f(len(b), a.ctypes.data, x.ctypes.data, b.ctypes.data, r.ctypes.data)
        return r

    return call


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -105], ids=["", "diagonal_below_range"])
@pytest.mark.parametrize("n,count", [(3, 60), (40, 30), (64, 20), (130, 10), (200, 6), (232, 4), (233, 4), (250, 4)])
def test_corrections_are_the_oracles(ctx, pkg, oracle_mod, residual, n, count, scale):
    """The FP32 factors and solves behind the corrections: the oracle's FP32
    getrf and getrs (correctly rounded reciprocals and quotients), bit for bit.
    The condition number of 3e4 keeps the corrections from converging to the
    same bits whatever the factors are."""
    rng = np.random.default_rng(n)
    As, bs = [], []
    for _ in range(count):
        q1, q2 = (np.linalg.qr(rng.standard_normal((n, n)))[0] for _ in range(2))
        As.append(np.asfortranarray(q1 * np.logspace(0, -4.5, n) @ q2) * scale)
        bs.append(rng.standard_normal(n))
    xs, it, info = _solve(ctx, pkg, As, bs)
    assert (info == 0).all() and (it >= 1).all(), it
    for a, b, x, k in zip(As, bs, xs, it):
        LU, ipiv, _ = oracle_mod.getrf(a.astype(np.float32))
        want, r = np.zeros(n), b
        for c in range(k):
            if c:
                r = residual(a, want, b)
            s = 2.0 ** np.floor(np.log2(np.abs(r).max()))
            want = want + s * oracle_mod.getrs(LU, ipiv, (r / s).astype(np.float32)).astype(np.float64)
        assert np.array_equal(x, want), (np.abs(x - want).max(), k)
