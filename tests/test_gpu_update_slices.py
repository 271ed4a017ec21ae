"""The FP32 SIMT update's slices (fetched one ahead) at depths around 16 and 32 and
ragged tiles: every tile gives the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (33, 17, 15), (64, 64, 16), (65, 31, 17), (128, 129, 31), (130, 100, 32),
                                   (97, 200, 33), (200, 64, 64), (70, 70, 65)])
def test_fp32_update_tiles_agree(ctx, monkeypatch, m, n, k):
    rng = np.random.default_rng(m + 7 * n + k)
    A, B, C = (rng.standard_normal(s).astype(np.float32) for s in ((m, k), (k, n), (m, n)))
    outs = []
    for tile in ("128", "64", "32", "16"):
        monkeypatch.setenv("GBLU_GEMM_TILE", tile)
        outs.append(ctx.gemm_update(C, A, B, "fp32"))
    for o in outs[1:]:
        assert np.array_equal(o, outs[0])
    ref = C.astype(np.float64) - A.astype(np.float64) @ B.astype(np.float64)
    bound = 2 * (k + 2) * 2.0 ** -24 * (np.abs(A).astype(np.float64) @ np.abs(B) + np.abs(C))
    assert np.all(np.abs(outs[0] - ref) <= bound)
