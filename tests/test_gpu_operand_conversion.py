"""The one-launch conversion of both operands of the tensor-core update at its
edges: rows, columns and depths that are not whole tiles or packs, and FP16
column scales of zero, tiny and huge columns."""
import numpy as np
import pytest

from test_gpu_mixed import _fp16_scaled, _round_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["bf16", "fp16"])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (63, 3, 63), (64, 4, 64), (65, 5, 65), (129, 257, 68), (321, 130, 259),
                                   (256, 131, 7)])
def test_conversion_edges(ctx, prec, m, n, k):
    rng = np.random.default_rng(m + n + k)
    A = rng.uniform(-1, 1, size=(m, k)).astype(np.float32)
    B = rng.standard_normal((k, n)).astype(np.float32)
    B[:, 0] = 0.0
    if n > 2:
        B[:, 1] *= np.float32(1e-30)
        B[:, 2] *= np.float32(1e30)
    C = rng.standard_normal((m, n)).astype(np.float32)
    out = ctx.gemm_update(C, A, B, prec)
    if prec == "bf16":
        Ar, Br = _round_bf16(A), _round_bf16(B)
    else:
        Ar, Br = A.astype(np.float16).astype(np.float64), _fp16_scaled(B)
    ref = C.astype(np.float64) - Ar @ Br
    scale = np.abs(Ar) @ np.abs(Br) + np.abs(C)
    err = np.abs(out.astype(np.float64) - ref) / scale
    # FP32 accumulation of k products and the subtraction
    assert err.max() < 4 * (k + 2) * 2.0 ** -24, err.max()
