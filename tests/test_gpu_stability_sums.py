"""Stability sums of long chains: the sums by binade (a step of many rows at once) must equal
the reference's row-by-row FP32 sum bit for bit, at the chain lengths where the work changes
hands, with ties in the rounding, with lambdas of zero-weight edges and with rows that change
the sum's binade at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chain(n, weights, oracle):
    """Two groups whose points join one by one in the order of their edges, then each other."""
    h = n // 3
    e = np.zeros(n - 1, oracle.MST_EDGE)
    e["from_node"] = np.arange(n - 1)
    e["to_node"] = np.arange(1, n)
    w = np.sort(weights.astype(np.float32))
    order = np.concatenate([np.arange(h - 1), np.arange(h, n - 1), [h - 1]])  # the link last
    e = e[order]
    e["weight"][:h - 1] = w[np.linspace(0, n - 3, h - 1).astype(int)]
    e["weight"][h - 1:-1] = w[np.linspace(0, n - 3, n - 1 - h).astype(int)]
    e["weight"][-1] = w[-1] * 2 + 1
    return oracle.sort_edges(e)


def _weights(kind, m, rng):
    if kind == "random":
        return rng.uniform(0.01, 2.0, m)
    if kind == "halves":  # lambda = j + 1/2: ties once the sum is above 2^23
        return 1.0 / (rng.integers(500, 3000, m) + 0.5)
    if kind == "zeros":
        w = rng.uniform(0.5, 2.0, m)
        w[: m // 2] = 0.0
        return w
    return 10.0 ** rng.uniform(-12, 12, m)  # "wide"


@pytest.mark.parametrize("kind", ["random", "halves", "zeros", "wide"])
@pytest.mark.parametrize("n", [40, 1000, 6150, 12300, 40011])
def test_long_chain_sums(ctx, oracle, n, kind):
    import torch
    from gpu_hdbscan_b200 import HDB_STAB_FP64
    mst = _chain(n, _weights(kind, n - 1, np.random.default_rng(n)), oracle)
    hier = oracle.linkage_tree(mst, n)
    h = torch.from_numpy(hier.view(np.int32).reshape(-1, 4).copy()).cuda()
    for mpts in (2, 5):
        cond = oracle.condensed_tree(hier, n, mpts)
        stab, s64 = oracle.stability(cond)
        for mode, ref in ((0, None), (HDB_STAB_FP64, s64)):
            labels, ncl, _, gstab = ctx.get_clusters(h, n, mpts, stability=mode, want_tree=True)
            got = gstab.cpu().numpy().copy().view(oracle.STABILITY).reshape(-1)
            np.testing.assert_array_equal(got["lambda"].view(np.uint32), stab["lambda"].view(np.uint32))
            rl, rn = oracle.get_clusters(cond, stab, n, ref)
            assert ncl == rn
            np.testing.assert_array_equal(labels.cpu().numpy(), rl)
