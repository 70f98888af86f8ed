"""The FP32 joins on given sample lists: every candidate they offer, against a restatement on the
CPU.  Points lie on an integer grid, where the FP32 sums are exact, so equal distances (the least
id counts) are everywhere; and the candidates' grouping by row, at the numbers of rows where the
buckets' size or the number of radix passes changes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

INF = np.float32(np.inf)


def _lists(n, m, S, rng, spread=None):
    """m sample lists of all kinds of sizes, with repeats of forward samples among the reverse
    ones, of old samples among the new ones, and more reverse samples offered than kept."""
    newS, oldS = np.zeros((m, 2 * S), np.int32), np.zeros((m, 2 * S), np.int32)
    counts = np.zeros((m, 4), np.int32)
    sizes = sorted({0, 1, min(2, S), S // 2, S})
    pool = np.arange(n) if spread is None else spread
    for j in range(m):
        nf, nr, of, orv = rng.choice(sizes, 4)
        ids = rng.choice(pool, min(4 * S, len(pool)), replace=False)
        ids = np.resize(ids, 4 * S)
        newS[j], oldS[j] = ids[:2 * S], ids[2 * S:]
        if j % 3 == 1:  # repeats: a reverse sample that is a forward one, a new one that is old
            newS[j, S] = newS[j, 0]
            oldS[j, 2 * S - 1] = oldS[j, 0]
            newS[j, S - 1] = oldS[j, S - 1]
        counts[j] = nf, of, nr + (7 if nr == S and j % 2 else 0), orv + (9 if orv == S else 0)
    return newS, oldS, counts


def _slots(row, fwd, rev, S):
    ids = np.concatenate([row[:fwd], row[S:S + min(rev, S)]])
    _, first = np.unique(ids, return_index=True)
    return ids[np.sort(first)]


def _offers(X, newS, oldS, counts, worst, cross_only):
    """Sorted (target, distance bits << 32 | id) of the reference's join of every list."""
    S = newS.shape[1] // 2
    out = []

    def offer(targets, ids, D):
        """to each target (row of D) the nearest of the ids (columns), the least id of those"""
        if not len(targets) or not len(ids):
            return
        key = D.astype(np.float32).view(np.uint32).astype(np.uint64) << np.uint64(32) | ids.astype(np.uint64)
        key = np.where(np.isinf(D), np.uint64(2**64 - 1), key)
        best = key.min(1)
        for t, b in zip(targets, best):
            if b != np.uint64(2**64 - 1) and np.uint32(b >> np.uint64(32)).view(np.float32) < worst[t]:
                out.append((int(t), int(b)))

    for j in range(len(newS)):
        nf, of, nr, orv = counts[j]
        new, old = _slots(newS[j], nf, nr, S), _slots(oldS[j], of, orv, S)
        new = new[~np.isin(new, old)]
        if not len(new) or len(new) + len(old) < 2 or (cross_only and not len(old)):
            continue
        A, B = X[new].astype(np.float64), X[old].astype(np.float64)
        if not cross_only:
            D = ((A[:, None] - A[None]) ** 2).sum(-1)
            np.fill_diagonal(D, np.inf)
            offer(new, new, D)
        D = ((A[:, None] - B[None]) ** 2).sum(-1)
        offer(new, old, D)
        offer(old, new, D.T)
    return sorted(out)


def _got(start, key):
    start, key = start.cpu().numpy().view(np.uint32).astype(np.int64), key.cpu().numpy().view(np.uint64)
    assert start[0] == 0 and (np.diff(start) >= 0).all()
    rows = np.repeat(np.arange(len(start) - 1), np.diff(start))
    return sorted(zip(rows.tolist(), key.tolist()))


@pytest.mark.parametrize("cross_only", [False, True])
@pytest.mark.parametrize("S", [1, 3, 4, 8, 16])
@pytest.mark.parametrize("d,form", [(1, 1), (4, 1), (5, 1), (12, 1), (17, 1), (28, 1), (2, 2), (12, 2), (28, 2),
                                    (29, 2), (32, 2), (33, 2), (64, 2), (101, 2)])
def test_candidates(ctx, d, form, S, cross_only):
    rng = np.random.default_rng(100 * d + S)
    n = 300
    X = rng.integers(0, 3, size=(n, d)).astype(np.float32)
    newS, oldS, counts = _lists(n, 400, S, rng)
    worst = rng.integers(1, 2 * d + 2, n).astype(np.float32)
    worst[rng.random(n) < 0.5] = INF
    ctx.set_join_tiles(form)
    try:
        got = ctx.fp32_join_candidates(X, newS, oldS, counts, worst, cross_only)
    finally:
        ctx.set_join_tiles(0)
    assert _got(*got) == _offers(X, newS, oldS, counts, worst, cross_only)


# one pass of the grouping up to 511 buckets of 256 rows, two with 128 rows a bucket and then 256,
# three past 2^26 - 256
@pytest.mark.parametrize("n", [511 * 256, 511 * 256 + 1, (1 << 25) - 128, (1 << 25) - 127, 1 << 25,
                               (1 << 26) - 256, (1 << 26) - 255])
def test_candidates_of_many_rows(ctx, n):
    import torch
    rng = np.random.default_rng(n)
    pool = np.unique(np.concatenate([rng.integers(0, n, 300), np.arange(20), n - 1 - np.arange(20),
                                     np.arange(120, 136), n - n % 256 - 1 - np.arange(10)]))
    X = torch.zeros((n, 2), device="cuda")
    x = rng.integers(0, 5, size=(len(pool), 2)).astype(np.float32)
    X[torch.from_numpy(pool).cuda()] = torch.from_numpy(x).cuda()
    newS, oldS, counts = _lists(n, 600, 8, rng, spread=pool)
    worst = torch.full((n,), float("inf"), device="cuda")
    start, key = ctx.fp32_join_candidates(X, newS, oldS, counts, worst)
    at = {int(p): i for i, p in enumerate(pool)}
    local = lambda a: np.vectorize(at.__getitem__)(a).astype(np.int32)
    ref = _offers(x, local(newS), local(oldS), counts, np.full(len(pool), INF), False)
    # local numbers follow the order of the rows, so the least local id is the least id
    ref = sorted((int(pool[t]), b >> 32 << 32 | int(pool[b & 0xffffffff])) for t, b in ref)
    start = start.cpu().numpy().view(np.uint32)
    assert start[0] == 0 and start[-1] == len(ref) and (start[1:] >= start[:-1]).all()
    rows = np.flatnonzero(start[1:] != start[:-1])
    key = key.cpu().numpy().view(np.uint64)
    assert sorted((int(r), int(k)) for r in rows for k in key[start[r]:start[r + 1]]) == ref


def test_lists_are_checked(ctx):
    from gpu_hdbscan_b200 import HdbError
    X, worst = np.zeros((10, 3), np.float32), np.full(10, INF)
    new, old = np.zeros((2, 4), np.int32), np.zeros((2, 4), np.int32)
    new[1, 2] = 10
    counts = np.array([[1, 1, 0, 0], [0, 0, 1, 0]], np.int32)
    with pytest.raises(HdbError, match="id outside"):
        ctx.fp32_join_candidates(X, new, old, counts, worst)
    counts[1] = 3, 0, 0, 0
    with pytest.raises(HdbError, match="count outside"):
        ctx.fp32_join_candidates(X, new, old, counts, worst)
