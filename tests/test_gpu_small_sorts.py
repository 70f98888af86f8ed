"""Sorts that run in one block (up to 8,192 items), at the sizes where the items per thread or the
path change: stable, with equal keys, keys that differ in one digit only, and negative ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["ties", "random", "one_digit", "equal"])
@pytest.mark.parametrize("m", [2, 31, 33, 255, 1023, 1024, 1025, 4097, 8191, 8192, 8193])
def test_sort_edges(ctx, oracle, m, kind):
    import torch
    rng = np.random.default_rng(m)
    e = np.zeros(m, oracle.MST_EDGE)
    e["from_node"] = np.arange(m)
    e["to_node"] = rng.integers(0, 1 << 20, m)
    if kind == "ties":
        e["weight"] = rng.integers(-9, 9, m).astype(np.float32) / 8
    elif kind == "random":
        e["weight"] = rng.normal(size=m) * 10.0 ** rng.integers(-6, 6, m)
    elif kind == "one_digit":
        e["weight"] = (np.float32(1.0).view(np.uint32) + rng.integers(0, 200, m).astype(np.uint32) * 256).view(np.float32)
    else:
        e["weight"] = 2.5
    ref = oracle.sort_edges(e)
    t = torch.from_numpy(e.view(np.int32).reshape(m, 3).copy()).cuda()
    got = ctx.sort_edges(t).cpu().numpy().copy().view(oracle.MST_EDGE).reshape(-1)
    np.testing.assert_array_equal(got, ref)
