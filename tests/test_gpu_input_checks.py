"""Inputs that are wrong, or not ready yet, when a call is made: neighbour ids outside the
point set are refused before anything is gathered through them, and a call waits for the
torch work that makes its arguments."""
import numpy as np
import pytest

from conftest import blobs

pytestmark = pytest.mark.gpu


def _ring(n, k):
    return ((np.arange(n)[:, None] + 1 + np.arange(k)) % n).astype(np.int32)


@pytest.mark.parametrize("bad", [-7, 500, 1 << 29])
def test_ids_outside_the_set_are_refused(ctx, bad):
    import torch
    from gpu_hdbscan_b200 import HdbError
    n, k = 500, 8
    X, ids = blobs(n, 5, 3), _ring(n, k)
    ids[123, k - 1] = bad
    with pytest.raises(HdbError, match="outside"):
        ctx.fix_distances(X, ids)
    label = -bad - 1 if bad < 0 else bad  # negative labels are old entries: the id is 6
    if bad < 0:
        return
    G = np.zeros((n, k, 2), np.int32)
    G[..., 1] = ids
    G[123, k - 1, 1] = label
    with pytest.raises(HdbError, match="outside"):
        ctx.hdbscan_from_knn(torch.from_numpy(G).cuda(), torch.from_numpy(X).cuda(), k=k, mpts=4)


def test_a_call_waits_for_its_arguments(ctx, oracle):
    import torch
    n, k = 4000, 8
    X = blobs(n, 12, 4)
    ids = _ring(n, k)
    want = oracle.fix_distances(X, ids)
    Xd = torch.from_numpy(X).cuda()
    made = torch.from_numpy(np.roll(ids, 1, axis=0)).cuda()  # valid ids, other rows'
    final = torch.from_numpy(ids).cuda()
    busy = torch.randn(8192, 8192, device="cuda")
    torch.cuda.synchronize()
    for _ in range(4):
        busy = busy @ busy
    made.copy_(final)
    got = ctx.fix_distances(Xd, made)
    np.testing.assert_array_equal(got.cpu().numpy().view(np.uint32), want.view(np.uint32))
