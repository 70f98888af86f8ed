"""The FP32 join in tiles of 4 rows x 1 to 8 columns: sample counts that take one column a
lane up to two passes over the rows, and numbers of dimensions around the staged chunks (a
chunk is 32) and the 16-byte pieces.  On an integer grid the sums are exact in FP32, so the
distances must equal the true ones and every row must be sorted by (distance, id)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,S", [(2, 1), (6, 3), (16, 8), (32, 16)])
@pytest.mark.parametrize("d", [29, 31, 32, 33, 36, 64, 65, 100])
def test_distances_on_a_grid(ctx, oracle, d, k, S):
    rng = np.random.default_rng(d + k)
    n = 600
    X = rng.integers(0, 4, size=(n, d)).astype(np.float32)
    D = ((X[:, None] - X[None]) ** 2).sum(-1)
    ids, dist = (a.cpu().numpy() for a in ctx.knn_split(
        ctx.NNDescent(X, k=k, sample_num=S, iterations=8)))
    assert oracle.validate_knn(ids)
    assert np.array_equal(dist, np.take_along_axis(D, ids.astype(np.int64), 1))
    key = dist.astype(np.float64) * n + ids
    assert (np.diff(key, axis=1) > 0).all()
    # as near as the oracle's graph on the whole.  Two runs differ in their reverse samples:
    # entries by some 20 %, so the sum of at least 1,200 by 0.6 %, two sums by 0.8 %; six of that
    oids, _ = oracle.nndescent(X, k, S, 8)
    ref = np.take_along_axis(D, np.asarray(oids).astype(np.int64), 1).sum()
    assert dist.sum() <= 1.05 * ref
