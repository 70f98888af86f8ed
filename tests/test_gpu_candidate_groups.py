"""Grouping of the join's candidates by target row: sizes at which the rows per bucket, the
number of radix passes or the last bucket's fill change.  A candidate that was lost or given to
another row would cost recall or leave a wrong distance in a row."""
import numpy as np
import pytest

from conftest import blobs

pytestmark = pytest.mark.gpu

# 511 full buckets of 8 and of 256 rows are the most that one 9-bit digit holds beside the one
# of the unused slots
SIZES = [9, 17, 511 * 8, 511 * 8 + 1, 511 * 16 - 3, 511 * 256, 511 * 256 + 1]


@pytest.mark.parametrize("n", SIZES)
def test_graph_is_the_reference_algorithms(ctx, oracle, n):
    k, S = 8, 4
    X = blobs(n, 6, seed=n, blobs=4)
    q = np.arange(0, n, max(1, n // 2000))
    gt, _ = oracle.bruteforce_knn(X, k, q)
    oids, _ = oracle.nndescent(X, k, S, 8)
    ids, dist = (a.cpu().numpy() for a in ctx.knn_split(
        ctx.NNDescent(X, k=k, sample_num=S, iterations=8)))
    assert oracle.validate_knn(ids)
    assert (np.diff(dist, axis=1) >= 0).all()
    # 0.5 points, and what one neighbour more or less of the sampled rows is
    assert oracle.recall(ids[q], gt, k) >= oracle.recall(oids[q], gt, k) - 0.005 - 1.0 / len(q)
    for i in np.random.default_rng(1).choice(n, min(n, 200), replace=False):
        for j in range(k):
            ref = np.float32(oracle.diffsum(X[i], X[ids[i, j]]))
            assert ref.view(np.uint32) == dist[i, j].view(np.uint32)
