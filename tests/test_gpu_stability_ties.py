"""Stability sums where additions are ties in the rounding by the thousand, and where the sum
does not move: lambdas that equal the birth, and infinite ones."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chains(na, nb, weights, link, oracle):
    """Two groups whose points join one by one, then each other at the weight `link`."""
    n = na + nb
    e = np.zeros(n - 1, oracle.MST_EDGE)
    order = np.concatenate([np.arange(na - 1), np.arange(na, n - 1), [na - 1]])  # the link last
    e["from_node"], e["to_node"] = order, order + 1
    e["weight"][:na - 1] = np.sort(weights[:na - 1])
    e["weight"][na - 1:-1] = np.sort(weights[na - 1:n - 2])
    e["weight"][-1] = link
    return oracle.sort_edges(e), n


def _exact_weights(m, lo, hi, part, rng):
    """Weights whose FP32 reciprocals are exactly j + 1/part, j in [lo, hi)."""
    lam = np.float32(np.arange(lo, hi) + 1.0 / part)
    w = (1.0 / lam.astype(np.float64)).astype(np.float32)
    w = w[(1.0 / w.astype(np.float64)).astype(np.float32) == lam]
    return rng.choice(w, m)


def _ties(rows, birth):
    """Ties among a cluster's additions, added up one by one."""
    s, ties = np.float32(0), 0
    for lam, size in zip(rows["lambda_val"], rows["child_size"]):
        y = np.float32(np.float32(lam - birth) * np.float32(size))
        if s > 0:
            x = float(y) / float(np.spacing(s))
            ties += x - np.floor(x) == 0.5 and s + y < 2 * s
        s = np.float32(s + y)
    return ties


def _compare(ctx, oracle, mst, n, mpts):
    import torch
    from gpu_hdbscan_b200 import HDB_STAB_FP32, HDB_STAB_FP64
    hier = oracle.linkage_tree(mst, n)
    cond = oracle.condensed_tree(hier, n, mpts)
    stab, s64 = oracle.stability(cond)
    h = torch.from_numpy(hier.view(np.int32).reshape(-1, 4).copy()).cuda()
    for mode, ref in ((HDB_STAB_FP32, None), (HDB_STAB_FP64, s64)):
        labels, ncl, _, gstab = ctx.get_clusters(h, n, mpts, stability=mode, want_tree=True)
        got = gstab.cpu().numpy().copy().view(oracle.STABILITY).reshape(-1)
        np.testing.assert_array_equal(got["lambda"].view(np.uint32), stab["lambda"].view(np.uint32))
        rl, rn = oracle.get_clusters(cond, stab, n, ref)
        assert ncl == rn
        np.testing.assert_array_equal(labels.cpu().numpy(), rl)
    return cond


# chains on both sides of the 4,096 nodes at which a block takes a chain
@pytest.mark.parametrize("na,nb,lo,hi", [(3900, 4090, 3000, 5000), (4097, 4098, 3000, 5000),
                                         (13000, 27000, 500, 3000)])
@pytest.mark.parametrize("part", [2, 4])
def test_thousands_of_ties(ctx, oracle, na, nb, lo, hi, part):
    rng = np.random.default_rng(na + part)
    # birth 1: the addends are j - 1 + 1/part, ties in the binade of the sum whose ulp is 2/part
    mst, n = _chains(na, nb, _exact_weights(na + nb, lo, hi, part, rng), 1.0, oracle)
    cond = _compare(ctx, oracle, mst, n, 2)
    for child in cond[cond["parent"] == n]["child"]:
        assert _ties(cond[cond["parent"] == child], np.float32(1.0)) >= 500


@pytest.mark.parametrize("na,nb", [(20, 33), (700, 4000), (4100, 9000)])
@pytest.mark.parametrize("kind", ["birth", "infinite", "half_infinite"])
def test_sums_that_stay(ctx, oracle, na, nb, kind):
    w = np.random.default_rng(nb).uniform(0.5, 1.0, na + nb).astype(np.float32)
    if kind == "birth":
        w[:] = 1.0
    else:
        w[: len(w) if kind == "infinite" else len(w) // 2] = 1e-42  # 1 / w is above FP32's range
        w = np.random.default_rng(na).permutation(w)
    mst, n = _chains(na, nb, w, 1.0, oracle)
    _compare(ctx, oracle, mst, n, 5)


@pytest.mark.parametrize("scale", [30, 36, -30])
def test_sums_at_the_ends_of_the_range(ctx, oracle, scale):
    """Weights near 1e30 make sums whose ulp is subnormal, with many points at once."""
    rng = np.random.default_rng(scale + 40)
    n = 20_000
    e = np.zeros(n - 1, oracle.MST_EDGE)
    e["to_node"] = np.arange(1, n)
    e["from_node"] = np.maximum(0, np.arange(n - 1) - rng.integers(0, 3, n - 1))
    e["weight"] = 10.0 ** (scale + rng.uniform(-2, 2, n - 1))
    for mpts in (2, 36):
        _compare(ctx, oracle, oracle.sort_edges(e), n, mpts)


def test_sums_that_stay_cost_no_more(ctx, oracle):
    """One by one they took over twenty times as long as sums that move."""
    import torch
    n, times = 1 << 20, []
    for w in (np.random.default_rng(0).uniform(0.5, 1.0, n).astype(np.float32), np.ones(n, np.float32)):
        mst, _ = _chains(n // 2, n // 2, w, 1.0, oracle)
        h = torch.from_numpy(oracle.linkage_tree(mst, n).view(np.int32).reshape(-1, 4).copy()).cuda()
        best = np.inf
        for _ in range(5):
            torch.cuda.synchronize()
            t = time.perf_counter()
            ctx.get_clusters(h, n, 2)
            best = min(best, time.perf_counter() - t)
        times.append(best)
    assert times[1] <= 4 * times[0]
