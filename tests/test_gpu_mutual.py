"""Mutual flags, reverse entries, in-degrees and id checks of the enhanced kNN graph: rows of
every load width (16, 8 and 4 bytes, by k and by where the ids start), rows that all list one
point, and each kind of bad row.  The graph must equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ids(n, k, seed):
    """Rows of k distinct other points, half of them near in the numbering; point 3 in most rows."""
    rng = np.random.default_rng(seed)
    out = np.empty((n, k), np.int32)
    for i in range(n):
        near = [(i + o) % n for o in range(1, k)] + [(i - o) % n for o in range(1, k)]
        pool = [3] + list(rng.permutation(near)[: k // 2]) + list(rng.choice(n, 3 * k))
        row = [v for v in dict.fromkeys(pool) if v != i][:k]
        out[i] = rng.permutation(row)
    return out


@pytest.mark.parametrize("k", [1, 2, 3, 4, 6, 8, 15, 16, 28, 30, 31, 32])
@pytest.mark.parametrize("start", [0, 1, 2])
def test_graph_of_any_rows(ctx, oracle, k, start):
    import torch
    n, d = 517, 4
    ids = _ids(n, k, 100 * k + start)
    X = np.random.default_rng(k).normal(size=(n, d)).astype(np.float32)
    dist = np.sqrt(((X[:, None] - X[ids]) ** 2).sum(-1)).astype(np.float32)
    nindex, nlist, ew, ah = oracle.enhanced_knng(ids, dist, X)
    t = torch.empty(n * k + 4, dtype=torch.int32, device="cuda")  # rows that start `start` ids in
    t[start:start + n * k] = torch.from_numpy(ids.reshape(-1)).cuda()
    g = ctx.buildEnhancedKNNG(t[start:start + n * k].view(n, k), dist, X)
    got = [a.cpu().numpy() for a in (g.nindex, g.nlist, g.eweight, g.antihubs)]
    assert np.array_equal(got[0], nindex) and np.array_equal(got[1], nlist)
    assert np.array_equal(got[2].view(np.uint32), ew.view(np.uint32))
    assert np.array_equal(np.sort(got[3]), np.sort(ah))


@pytest.mark.parametrize("k", [3, 6, 32])
@pytest.mark.parametrize("bad,match", [("high", "outside"), ("low", "outside"), ("self", "own id"), ("twice", "repeats")])
def test_bad_rows_are_refused(ctx, k, bad, match):
    n = 300
    ids = _ids(n, k, k)
    X = np.random.default_rng(k).normal(size=(n, 3)).astype(np.float32)
    dist = np.ones((n, k), np.float32)
    r, c = 217, k - 1
    ids[r, c] = {"high": n, "low": -1 - c, "self": r, "twice": ids[r, 0]}[bad]
    with pytest.raises(Exception, match=match):
        ctx.buildEnhancedKNNG(ids, dist, X)
