"""The kernels that gather whole rows for exact difference sums (the initial graph and the
FP32 re-rank): copies of 4, 2 and 1 floats, dimensions around the staged chunk of 64, and
neighbour counts that leave lanes idle.  Distances must equal the sequential FP32 sum bit for
bit."""
import numpy as np
import pytest

from conftest import blobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,k", [(1, 3), (2, 32), (3, 17), (4, 5), (6, 8), (31, 32), (33, 20), (63, 31), (64, 32),
                                 (65, 16), (66, 24), (68, 32), (127, 7), (128, 32), (130, 32), (201, 12)])
@pytest.mark.parametrize("precision,iterations", [(0, 0), (1, 1)])
def test_distance_bits(ctx, oracle, d, k, precision, iterations):
    n = 700
    X = blobs(n, d, seed=d + k, blobs=5)
    ids, dist = (a.cpu().numpy() for a in ctx.knn_split(
        ctx.NNDescent(X, k=k, sample_num=k // 2, iterations=iterations, precision=precision)))
    assert oracle.validate_knn(ids)
    for i in range(0, n, 9):
        for j in range(k):
            ref = np.float32(oracle.diffsum(X[i], X[ids[i, j]]))
            assert ref.view(np.uint32) == dist[i, j].view(np.uint32)
