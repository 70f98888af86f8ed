"""The FP32 join of short rows (d <= 28): every number of 16-byte pieces, aligned or not, and
sample counts that make the warp work on one, two or four parts.  Its graph must reach the
reference algorithm's recall with exact distances, as the tile forms' does; with many equal
distances (integer coordinates) every row must be sorted by (distance, id)."""
import numpy as np
import pytest

from conftest import blobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 3, 4, 7, 8, 11, 12, 16, 17, 20, 23, 24, 28, 29])
def test_recall_and_distances(ctx, oracle, d):
    n, k, S = 3000, 24, 12
    X = blobs(n, d, seed=d, blobs=4)
    q = np.arange(0, n, 3)
    gt, _ = oracle.bruteforce_knn(X, k, q)
    oids, _ = oracle.nndescent(X, k, S, 6)
    ids, dist = (a.cpu().numpy() for a in ctx.knn_split(
        ctx.NNDescent(X, k=k, sample_num=S, iterations=6)))
    assert oracle.validate_knn(ids)
    assert oracle.recall(ids[q], gt, k) >= oracle.recall(oids[q], gt, k) - 0.005
    for i in np.random.default_rng(1).choice(n, 60, replace=False):
        for j in range(k):
            ref = np.float32(oracle.diffsum(X[i], X[ids[i, j]]))
            assert ref.view(np.uint32) == dist[i, j].view(np.uint32)


@pytest.mark.parametrize("k,S", [(2, 1), (4, 2), (8, 4), (16, 8), (32, 16)])
@pytest.mark.parametrize("d", [2, 5, 12])
def test_equal_distances(ctx, k, S, d):
    """A small set on an integer grid, in every form: exact distances, rows by (distance, id)."""
    rng = np.random.default_rng(10 * k + d)
    n = 2 * k + 5
    X = rng.integers(0, 3, size=(n, d)).astype(np.float32)
    D = ((X[:, None] - X[None]) ** 2).sum(-1)
    got = {}
    for tiles in (0, 1, 2):
        ctx.set_join_tiles(tiles)
        ids, dist = (a.cpu().numpy() for a in ctx.knn_split(
            ctx.NNDescent(X, k=k, sample_num=S, iterations=40)))
        got[tiles] = (ids, dist)
    ctx.set_join_tiles(0)
    for ids, dist in got.values():
        assert np.array_equal(dist, np.take_along_axis(D, ids.astype(np.int64), 1))
        key = dist.astype(np.float64) * n + ids
        assert (np.diff(key, axis=1) > 0).all()
