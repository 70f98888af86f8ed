"""Trees above the sizes at which the work leaves one block's shared memory: linkage levels
outside the blocks of 2,048 ranks, and more than 8,192 splits and clusters in the condensed tree."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _random_tree(n, oracle, tied, seed):
    """A random spanning tree, its edges sorted by their random weights."""
    rng = np.random.default_rng(seed)
    e = np.zeros(n - 1, oracle.MST_EDGE)
    e["to_node"] = np.arange(1, n)
    e["from_node"] = rng.integers(0, np.arange(1, n))
    p = rng.permutation(n).astype(np.int32)
    e["to_node"], e["from_node"] = p[e["to_node"]], p[e["from_node"]]
    e["weight"] = rng.integers(1, 400, n - 1) / 64.0 if tied else rng.uniform(0.01, 2.0, n - 1)
    return oracle.sort_edges(e)


@pytest.mark.parametrize("tied", [False, True])
@pytest.mark.parametrize("edges", [2048, 2049, 4097, 303_104, 303_105, 700_001, 1 << 20])
def test_linkage_tree(ctx, oracle, edges, tied):
    import torch
    n = edges + 1
    mst = _random_tree(n, oracle, tied, edges)
    ref = oracle.linkage_tree(mst, n)
    t = torch.from_numpy(mst.view(np.int32).reshape(-1, 3).copy()).cuda()
    got = ctx.build_Linkage_tree(t, n).cpu().numpy().copy().view(oracle.LINKAGE_NODE).reshape(-1)
    np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("tied", [False, True])
@pytest.mark.parametrize("n,mpts", [(30_000, 2), (100_000, 2), (400_000, 5)])
def test_clusters(ctx, oracle, n, mpts, tied):
    import torch
    from gpu_hdbscan_b200 import HDB_STAB_FP32, HDB_STAB_FP64
    hier = oracle.linkage_tree(_random_tree(n, oracle, tied, n), n)
    cond = oracle.condensed_tree(hier, n, mpts)
    stab, s64 = oracle.stability(cond)
    assert len(stab) > 8192
    rows = cond[np.lexsort((cond["child"], cond["parent"]))]  # the order of the library's rows
    h = torch.from_numpy(hier.view(np.int32).reshape(-1, 4).copy()).cuda()
    for mode, ref in ((HDB_STAB_FP32, None), (HDB_STAB_FP64, s64)):
        labels, ncl, gcond, gstab = ctx.get_clusters(h, n, mpts, stability=mode, want_tree=True)
        np.testing.assert_array_equal(
            gcond.cpu().numpy().copy().view(oracle.CONDENSED_NODE).reshape(-1), rows)
        np.testing.assert_array_equal(
            gstab.cpu().numpy().copy().view(oracle.STABILITY).reshape(-1)["lambda"].view(np.uint32),
            stab["lambda"].view(np.uint32))
        rl, rn = oracle.get_clusters(cond, stab, n, ref)
        assert ncl == rn
        np.testing.assert_array_equal(labels.cpu().numpy(), rl)
