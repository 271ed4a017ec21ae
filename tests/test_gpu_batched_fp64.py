"""The FP64 batch's update tiles (groups of 8 rows and 4 columns) and its
reciprocals at their edges, bit for bit against the oracle."""
import numpy as np
import pytest

from test_gpu_batched import Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e-308, 5e-320, 1e307])
def test_fp64_batch_edges_bit_exact(ctx, oracle_mod, scale):
    """Every remainder of rows and columns from a panel of 8 on; matrices scaled so
    that pivots or their reciprocals leave the normal numbers."""
    sizes = np.array(list(range(1, 50)) + [63, 64, 65, 72, 73, 95, 97, 127, 128, 129, 136, 137, 200, 233, 255, 256],
                     dtype=np.int64)
    rng = np.random.default_rng(7)
    A = np.concatenate([rng.uniform(-1, 1, n * n) for n in sizes]) * scale
    b = rng.standard_normal(int(sizes.sum()))
    bt = Batch(ctx, sizes, 0)
    X, info = bt.solve(A, b)
    _, Xref, info_ref = oracle_mod.gesv_batched(sizes, A, b)
    assert np.array_equal(info, info_ref)
    assert np.array_equal(X, Xref, equal_nan=True)
    bt.close()
