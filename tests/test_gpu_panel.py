"""The sub-panel cluster kernel (leaves of getrf) at the edges of its variants:
pivots and factors bit-identical to the oracle, whatever the number of CTAs,
chain warps, rows per thread and the leaf width a height gives."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (rows, columns): variant edges by height, ragged leaves and sub-panels,
# last CTAs with few or no rows
FP64_SHAPES = [(33, 33), (95, 64), (481, 70), (512, 65), (513, 72), (1024, 64), (1025, 71), (1300, 64),
               (2048, 33), (2049, 130), (4096, 64), (4097, 40), (8192, 32), (8193, 33)]
FP32_SHAPES = [(32, 32), (33, 33), (128, 128), (129, 129), (256, 200), (257, 130), (512, 128), (513, 140),
               (1024, 128), (1025, 131), (2048, 20), (2049, 256), (4096, 128), (4097, 70), (8192, 64),
               (8193, 33), (16384, 32), (16385, 40)]


def _sgetrf(lib, A):
    LU = np.array(A, order="F", copy=True)
    m, n = LU.shape
    ipiv = np.zeros(min(m, n), dtype=np.int64)
    m_, n_, lda, info = ctypes.c_int64(m), ctypes.c_int64(n), ctypes.c_int64(m), ctypes.c_int64()
    lib.gblu_sgetrf_(ctypes.byref(m_), ctypes.byref(n_), LU.ctypes.data, ctypes.byref(lda), ipiv.ctypes.data,
                     ctypes.byref(info))
    return LU, ipiv, info.value


def _check(pkg, oracle_mod, A):
    if A.dtype == np.float32:
        LU, ipiv, info = _sgetrf(pkg.load_library(), A)
    else:
        LU, ipiv, info = pkg.dgetrf(A)
    LUo, ipivo, infoo = oracle_mod.getrf(A)
    assert info == infoo
    assert np.array_equal(ipiv, ipivo)
    assert np.array_equal(LU, LUo, equal_nan=True)


@pytest.mark.parametrize("m,n", FP64_SHAPES)
def test_fp64_variants_bit_exact(pkg, oracle_mod, m, n):
    _check(pkg, oracle_mod, np.random.default_rng(m + 7 * n).standard_normal((m, n)))


@pytest.mark.parametrize("m,n", FP32_SHAPES)
def test_fp32_variants_bit_exact(pkg, oracle_mod, m, n):
    _check(pkg, oracle_mod, np.random.default_rng(m + 7 * n).standard_normal((m, n)).astype(np.float32))


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("m", [90, 300, 1300])
@pytest.mark.parametrize("kind", ["ties", "zero_columns", "nan", "tiny", "huge", "subnormal"])
def test_special_values(pkg, oracle_mod, dtype, m, kind):
    """Equal candidates, zero pivots, NaN, and pivots whose reciprocal leaves
    the range of the integer reciprocal (the division is used there)."""
    rng = np.random.default_rng(m)
    A = rng.standard_normal((m, 70)).astype(dtype)
    fi = np.finfo(dtype)
    if kind == "ties":
        A = rng.integers(-2, 3, size=(m, 70)).astype(dtype)
    elif kind == "zero_columns":
        A[:, [0, 9, 40]] = 0
    elif kind == "nan":
        A[m // 2, 5] = np.nan
    elif kind == "tiny":
        A *= fi.tiny * 4
    elif kind == "huge":
        A *= fi.max / 64
    else:
        A *= fi.tiny / 64
    _check(pkg, oracle_mod, A)


def test_integer_reciprocal_matches_ieee():
    """recip_normal gives RN(1 / x) bit for bit: every FP32 significand, 2^24
    FP64 operands (edge significands included)."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    lib = ctypes.CDLL(os.path.join(root, "linearsolve.jl_gb300", "libgblu_tools.so"))
    lib.gblu_tool_recipcheck.argtypes = [ctypes.c_int64, ctypes.c_uint64, ctypes.POINTER(ctypes.c_uint64),
                                         ctypes.POINTER(ctypes.c_uint64)]
    lib.gblu_tool_recipcheck.restype = ctypes.c_int32
    m64, m32 = ctypes.c_uint64(), ctypes.c_uint64()
    assert lib.gblu_tool_recipcheck(1 << 24, 99, ctypes.byref(m64), ctypes.byref(m32)) == 0
    assert m64.value == 0 and m32.value == 0, (m64.value, m32.value)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("m", [1, 31, 33, 63, 64, 65, 95, 127, 128, 130])
@pytest.mark.parametrize("extra", [1, 3, 700])
def test_wide_trsm_bit_exact(pkg, oracle_mod, dtype, m, extra):
    """U12 := L11 \\ A12 of a wide matrix: orders around the 32-row blocks, the
    16-byte and the element copies of L, few and many columns."""
    _check(pkg, oracle_mod, np.random.default_rng(m + extra).standard_normal((m, m + extra)).astype(dtype))


def test_newton_reciprocal_matches_ieee():
    """recip_rn gives 1 / x bit for bit on all 2^32 FP32 operands."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    lib = ctypes.CDLL(os.path.join(root, "linearsolve.jl_gb300", "libgblu_tools.so"))
    lib.gblu_tool_reciprncheck.argtypes = [ctypes.POINTER(ctypes.c_uint64)]
    lib.gblu_tool_reciprncheck.restype = ctypes.c_int32
    m = ctypes.c_uint64()
    assert lib.gblu_tool_reciprncheck(ctypes.byref(m)) == 0
    assert m.value == 0, m.value


def _panelcheck(A, at):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    f = ctypes.CDLL(os.path.join(root, "linearsolve.jl_gb300", "libgblu_tools.so")).gblu_tool_panelcheck
    f.argtypes = [ctypes.c_int32, ctypes.c_int64, ctypes.c_void_p, ctypes.c_int32] + 4 * [ctypes.c_void_p]
    f.restype = ctypes.c_int32
    A = np.array(A, order="F", copy=True)
    ipiv, moves = np.zeros(A.shape[1], dtype=np.int64), np.zeros((256, 2), dtype=np.int32)
    count, code = np.zeros(1, dtype=np.int32), np.zeros(1, dtype=np.int32)
    assert f(A.dtype == np.float64, A.shape[0], A.ctypes.data, at, ipiv.ctypes.data, moves.ctypes.data,
             count.ctypes.data, code.ctypes.data) == 0
    return A, ipiv, moves[: min(count[0], 256)], int(code[0])


@pytest.mark.parametrize("dtype,m", [(np.float64, 100), (np.float64, 512), (np.float32, 700)])
@pytest.mark.parametrize("at", [-1, 0, 40, 390, 775, 1000, 2600])
def test_late_push_gives_up_in_bounds(ctx, oracle_mod, dtype, m, at):
    """One CTA late with one of its pushes (a candidate or a moved row) by more
    than the wait limit: the launch ends with the error code, pivots and moves
    name rows of the leaf, and the context goes on.  Never late: the oracle's
    pivots and factors, and no code."""
    A = np.random.default_rng(m).standard_normal((m, 64 if dtype == np.float64 else 128)).astype(dtype)
    LU, ipiv, moves, code = _panelcheck(A, at)
    assert ((ipiv >= 1) & (ipiv <= m)).all()
    assert ((moves >= 0) & (moves < m)).all()
    if at < 0:
        LUo, ipivo, _ = oracle_mod.getrf(A)
        assert code == 0
        assert np.array_equal(ipiv, ipivo) and np.array_equal(LU, LUo)
    else:
        assert code == 1  # DEV_TIMEOUT_PANEL
    B = np.random.default_rng(0).standard_normal((300, 300))
    f = ctx.factor(300, 300)
    assert f.getrf(B) == 0
    assert np.array_equal(f.factors(), oracle_mod.getrf(B)[0])
    f.close()

