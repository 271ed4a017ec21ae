"""The 128-column no-pivot leaf of the butterfly-transformed factors at its
edges: ragged last leaves, sub-block boundaries, rows below the leaf around a
CTA's 32, and the trailing solves through the inverse the leaf leaves behind."""
import ctypes
from importlib import import_module

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


def _leaf(ctx, pkg, A, pad):
    """The leaf's two launches on A (m x w, FP32) as they are given to it."""
    rt = import_module(pkg.__name__ + "._cuda").runtime()
    m, w = A.shape
    lda = m + pad
    host = np.zeros((lda, w), dtype=np.float32, order="F")
    host[:m] = A
    ipiv, info = np.zeros(w, dtype=np.int64), np.zeros(1, dtype=np.int64)
    linv = np.zeros((128, 128), dtype=np.float32, order="F")
    bufs = []
    for x in (host, ipiv, info, linv, np.zeros(1 << 18, dtype=np.float32)):
        p = ctypes.c_void_p()
        assert rt.cudaMalloc(ctypes.byref(p), x.nbytes) == 0
        assert rt.cudaMemcpy(p, x.ctypes.data, x.nbytes, 1) == 0
        bufs.append(p)
    launch = ctx.lib._ZN4gblu17genp_panel_launchEPfllliPlS1_PvS0_P11CUstream_st
    launch.argtypes = ([ctypes.c_void_p] + 3 * [ctypes.c_int64] + [ctypes.c_int] + 5 * [ctypes.c_void_p])
    assert launch(bufs[0], lda, m, 0, w, bufs[1], bufs[2], bufs[4], bufs[3] if w == 128 else None, None) == 0
    for x, p in zip((host, ipiv, info, linv), bufs):
        assert rt.cudaMemcpy(x.ctypes.data, p, x.nbytes, 2) == 0
    for p in bufs:
        rt.cudaFree(p)
    assert np.array_equal(ipiv, np.arange(1, w + 1))
    assert not host[m:].any()
    return host[:m], int(info[0]), linv


@pytest.mark.parametrize("m,w,pad", [(128, 128, 0), (129, 128, 3), (160, 128, 0), (1000, 128, 1), (190, 97, 2), (70, 64, 0),
                                     (300, 33, 0), (40, 31, 0), (33, 1, 0)])
def test_leaf_is_substitution(ctx, pkg, m, w, pad):
    """|A - L U| <= 2 w u |L| |U| in every element, as for substitution whatever
    the condition of U's 32 x 32 diagonal blocks (here 1.6^31; an inverse of
    one leaves its condition times u)."""
    rng = np.random.default_rng(m + w)
    U = np.triu(rng.uniform(-0.05, 0.05, (w, w)), 1) + np.eye(w)
    for b in range(0, w, 32):
        s = slice(b, min(b + 32, w))
        k = s.stop - b
        U[s, s] = np.eye(k) - 0.6 * np.triu(np.ones((k, k)), 1)
    L = rng.uniform(-1, 1, (m, w))
    L[:w] = 0.1 * np.tril(L[:w], -1) + np.eye(w)
    A = (L @ U).astype(np.float32)
    F, info, linv = _leaf(ctx, pkg, A, pad)
    assert info == 0
    Fd = F.astype(np.float64)
    Lc = np.vstack([np.tril(Fd[:w], -1) + np.eye(w), Fd[w:]])
    Uc = np.triu(Fd[:w])
    assert (np.abs(A - Lc @ Uc) <= 2 * w * 2.0 ** -24 * (np.abs(Lc) @ np.abs(Uc))).all()
    if w == 128:  # the inverse of L11: |L X - I| <= 2 w u |L| |X| by columns
        X = linv.astype(np.float64)
        R = np.abs(Lc[:w] @ X - np.eye(w))
        assert (R <= 2 * w * 2.0 ** -24 * (np.abs(Lc[:w]) @ np.abs(X))).all()


@pytest.mark.parametrize("m", [128, 200])
@pytest.mark.parametrize("k", [0, 5, 31, 32, 40, 95, 127])
def test_leaf_zero_in_a_later_block(ctx, pkg, m, k):
    """A pivot that is exactly zero: info is its column, the column's
    multipliers stay unscaled, and the columns after it go on."""
    w = 128
    rng = np.random.default_rng(k)
    A = (rng.uniform(-1, 1, (m, w)) + 40 * np.eye(m, w)).astype(np.float32)
    A[k, : k + 1] = 0  # row k and column k take no update before step k
    A[:k, k] = 0
    F, info, _ = _leaf(ctx, pkg, A, 0)
    assert info == k + 1
    assert np.array_equal(F[k + 1:, k], A[k + 1:, k])
    assert F[k, k] == 0 and np.isfinite(F).all()
    Fd = F.astype(np.float64)
    Lc = np.vstack([np.tril(Fd[:w], -1) + np.eye(w), Fd[w:]])
    Uc = np.triu(Fd[:w])
    keep = np.arange(w) != k  # column k is not L U: its multipliers are not quotients
    R = np.abs(A - Lc @ Uc)[:, keep]
    assert (R <= 2 * w * 2.0 ** -24 * (np.abs(Lc) @ np.abs(Uc))[:, keep]).all()
