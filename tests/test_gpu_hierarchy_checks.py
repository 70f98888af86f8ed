"""Hierarchies that are no tree are refused: a node that two others name as their child, with
sizes that add up all the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _refused(ctx, h, n, mpts):
    import torch
    from gpu_hdbscan_b200 import HdbError
    with pytest.raises(HdbError, match="valid single-linkage tree"):
        ctx.get_clusters(torch.from_numpy(h).cuda(), n, mpts)


def test_an_internal_node_with_two_parents(ctx):
    n = 6  # nodes 6 = (0, 1), 7 = (6, 2), 8 = (6, 3), 9 = (7, 8), 10 = (9, 4)
    h = np.array([[0, 1, 0, 2], [6, 2, 0, 3], [6, 3, 0, 3], [7, 8, 0, 6], [9, 4, 0, 7]], np.int32)
    h[:, 2] = np.arange(1, 6, dtype=np.float32).view(np.int32)
    for mpts in (2, 3, 6):
        _refused(ctx, h, n, mpts)


@pytest.mark.parametrize("n", [5, 300, 5000])
def test_a_point_with_two_parents(ctx, oracle, n):
    import torch
    rng = np.random.default_rng(n)
    e = np.zeros(n - 1, oracle.MST_EDGE)
    e["to_node"] = np.arange(1, n)
    e["from_node"] = rng.integers(0, np.arange(1, n))
    e["weight"] = rng.uniform(0.1, 1.0, n - 1)
    good = oracle.linkage_tree(oracle.sort_edges(e), n).view(np.int32).reshape(-1, 4)
    ctx.get_clusters(torch.from_numpy(good.copy()).cuda(), n, 2)  # the tree itself is taken
    r, side = np.argwhere(good[:, :2] < n)[-1]
    for other in ((good[r, side] + 1) % n, (good[r, side] + n // 2) % n):
        h = good.copy()
        h[r, side] = other
        if h[r, 0] != h[r, 1]:
            _refused(ctx, h, n, 2)
