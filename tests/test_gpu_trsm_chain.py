"""TRSM of the 16-bit-operand factors through a chain of inverted 128-row blocks,
at its edges: triangles just above 64 rows, ragged last blocks, one to four
blocks, and more than a chain takes."""
import pytest

from test_gpu_mixed import _factor_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["bf16", "fp16"])
@pytest.mark.parametrize("n", [130, 193, 260, 388, 520, 641, 1030, 1100, 2180])
def test_chain_against_substitution(ctx, pkg, monkeypatch, prec, n):
    """As accurate as the substitution chain, whose updates have the same
    operands (or, inside a chain, FP32 ones)."""
    A, _ = pkg.workloads.plain(n, 1, seed=500 + n)
    e_inv, lmax, _ = _factor_error(ctx, monkeypatch, A, prec, "default", env="GBLU_TRSM")
    e_sub, _, _ = _factor_error(ctx, monkeypatch, A, prec, "exact", env="GBLU_TRSM")
    assert lmax <= 1.0
    assert e_inv < 2 * e_sub + 1e-3, (e_inv, e_sub)
