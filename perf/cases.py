"""The calls that users of this library make, as performance cases.

The library clusters vectors: NN-Descent kNN graph -> enhanced kNN graph -> MST ->
linkage tree -> condensed tree -> labels.  A case is one call (or one short sequence of
calls) of ``gpu_hdbscan_b200.Context``:

    knn     the kNN graph alone (NNDescent)
    run     the whole path on one point set (hdbscan), from device or from host memory
    batch   the whole path on many independent point sets at once (hdbscan_batched)
    tail    the stages after a finished kNN graph (hdbscan_from_knn)
    merge   the union of two kNN graphs (KNNMerge)
    stages  the stage functions one by one, with their other options: fix_distances,
            buildEnhancedKNNG, the three MST modes, sort_edges, build_Linkage_tree,
            get_clusters (64-bit stabilities, condensed tree), build_CoreSG

NN-Descent takes its samples in the order in which the GPU's threads happen to arrive, so
neighbour ids, and with them the numbering of the clusters, change from run to run.  What
is reproducible about its graph are the sorted neighbour distances of every row: the cases
that build a graph return those (Euclidean), whole.  The cases that start from a given
graph are exact: they return labels, trees and graphs.

Points are Gaussian blobs with 5 % uniform noise, the mixture of the repository's
benchmark, with 5 to 200 blobs and centres a few standard deviations apart.
"""
import math
import random
import weakref

import numpy as np
import torch

import gpu_hdbscan_b200 as hdb

_PRECISION = {"fp32": hdb.HDB_PREC_FP32, "bf16": hdb.HDB_PREC_BF16, "fp16": hdb.HDB_PREC_FP16}
_SPREAD = 2.0   # blob centres are uniform in [-_SPREAD, _SPREAD] in every dimension
_NOISE = 0.05
_ITERATIONS = 6
_MERGE_SAMPLES, _MERGE_ITERATIONS = 12, 11  # KNNMerge's defaults

_open = weakref.WeakValueDictionary()


def _context():
    """The program's one context; it lives as long as some state uses it."""
    device = torch.cuda.current_device()
    ctx = _open.get(device)
    if ctx is None:
        ctx = _open[device] = hdb.Context(device)
    return ctx


# ---- the cases -----------------------------------------------------------------
def listed():
    return [
        # exploring a small table: one short call, all launches and waits
        {"name": "knn_small_f32", "kind": "knn", "n": 1500, "d": 8, "k": 16, "precision": "fp32"},
        # the repository's 100k x 12 configuration, tensor-core form
        {"name": "knn_100k_bf16", "kind": "knn", "n": 100_000, "d": 12, "k": 32, "precision": "bf16"},
        # odd sizes: rows that are not 16-byte multiples, n and k not powers of two
        {"name": "knn_odd_f16", "kind": "knn", "n": 300_007, "d": 33, "k": 20, "precision": "fp16"},
        # embeddings in the reference arithmetic: the FP32 join at a large d
        {"name": "knn_wide_f32", "kind": "knn", "n": 200_000, "d": 128, "k": 32, "precision": "fp32"},
        # a small table from a user's host array, labels back on the host
        {"name": "run_host_f32", "kind": "run", "n": 5000, "d": 12, "k": 32, "precision": "fp32",
         "host": True},
        # an ordinary device-resident run
        {"name": "run_1m_bf16", "kind": "run", "n": 1_000_000, "d": 64, "k": 32, "precision": "bf16",
         "host": False},
        # the repository's 10M x 12 size in its FP32 form
        {"name": "run_10m_f32", "kind": "run", "n": 10_000_000, "d": 12, "k": 32,
         "precision": "fp32", "host": False},
        # the benchmark's size and form: 20M x 128, tensor cores
        {"name": "run_20m_bf16", "kind": "run", "n": 20_000_000, "d": 128, "k": 32,
         "precision": "bf16", "host": False},
        # many small independent clusterings, the batched workload's sizes and dimensions
        {"name": "batch_f32", "kind": "batch", "count": 96, "n_lo": 1000, "n_hi": 40_000,
         "dims": "8,12,32,64", "k": 16, "precision": "fp32"},
        # clustering again on a kept graph
        {"name": "tail_2m", "kind": "tail", "n": 2_000_000, "d": 16, "k": 32, "mpts": 32},
        # two shards' graphs joined
        {"name": "merge_f32", "kind": "merge", "n": 60_000, "n2": 100_003, "d": 12, "k": 32},
        # the stage interface, one function after the other
        {"name": "stages_150k", "kind": "stages", "n": 150_000, "d": 24, "k": 24, "mpts": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges, its cost at most that of the largest listed one."""
    kind = rng.choice(["knn", "knn", "run", "run", "batch", "tail", "merge", "stages"])
    if kind in ("knn", "run"):
        precision = rng.choice(["fp32", "bf16", "fp16"])
        d = rng.choice([8, 12, 13, 16, 24, 33, 50, 64, 96, 100, 128, 160, 256])
        k = rng.choice([16, 20, 24, 32, 32])
        # up to 1.5e8 coordinates in FP32, 1e9 on the tensor cores
        top = min(4_000_000, int((1.5e8 if precision == "fp32" else 1e9) / d))
        case = {"kind": kind, "n": _log(rng, 1000, top), "d": d, "k": k, "precision": precision}
        if kind == "run":
            case["host"] = case["n"] * d < 20_000_000 and rng.random() < 0.4
        return case
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(5, 150), "n_lo": _log(rng, 1000, 3000),
                "n_hi": _log(rng, 5000, 40_000), "dims": rng.choice(["8,12,32,64", "12", "16,33", "96"]),
                "k": rng.choice([16, 32]), "precision": rng.choice(["fp32", "bf16"])}
    if kind == "tail":
        k = rng.choice([12, 16, 24, 32])
        return {"kind": "tail", "n": _log(rng, 2000, 3_000_000), "d": rng.choice([8, 12, 17, 32, 64]),
                "k": k, "mpts": rng.choice([5, 8, k])}
    if kind == "merge":
        return {"kind": "merge", "n": _log(rng, 2000, 80_000), "n2": _log(rng, 2000, 80_000),
                "d": rng.choice([8, 12, 21, 32]), "k": rng.choice([24, 32])}
    k = rng.choice([12, 16, 24, 32])
    return {"kind": "stages", "n": _log(rng, 2000, 400_000), "d": rng.choice([8, 12, 19, 24, 48]),
            "k": k, "mpts": rng.choice([5, 10, k])}


# ---- inputs --------------------------------------------------------------------
def _blobs(n):
    return max(5, min(200, n // 10_000))


def _points(n, d, seed):
    """-> (X [n, d] float32 on the GPU, the blob of every row, -1 for noise)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    blobs = _blobs(n)
    centres = torch.empty((blobs, d), device="cuda").uniform_(-_SPREAD, _SPREAD, generator=g)
    sigma = torch.empty((blobs, 1), device="cuda").uniform_(0.7, 1.3, generator=g)
    which = torch.randint(0, blobs, (n,), device="cuda", generator=g)
    noise = torch.empty(n, device="cuda").uniform_(generator=g) < _NOISE
    X = torch.empty((n, d), device="cuda")
    step = max(1, (1 << 28) // d)
    for a in range(0, n, step):
        x, w = X[a:a + step], which[a:a + step]
        x.normal_(generator=g).mul_(sigma[w]).add_(centres[w])
        rows = noise[a:a + step].nonzero()[:, 0]
        x[rows] = torch.empty((rows.numel(), d), device="cuda").uniform_(
            -_SPREAD - 2, _SPREAD + 2, generator=g)
    which[noise] = -1
    return X, which


def _nearest(Q, X, k, skip=None):
    """The k nearest rows of X for every row of Q, nearest first -> (squared distances, ids);
    skip: the row of X that a row of Q is."""
    dist, ids = [], []
    xx = X.square().sum(1)
    step = max(1, (1 << 27) // X.shape[0])
    for a in range(0, Q.shape[0], step):
        q = Q[a:a + step]
        D = torch.addmm(xx[None, :] + q.square().sum(1)[:, None], q, X.T, alpha=-2)
        if skip is not None:
            D.scatter_(1, skip[a:a + step, None], float("inf"))
        v, i = D.topk(k, dim=1, largest=False)
        dist.append(v.clamp_(min=0))
        ids.append(i)
    return torch.cat(dist), torch.cat(ids)


def _knn(X, which, k):
    """A finished kNN graph of the points: every row's nearest neighbours among 8,192 rows of its
    blob or fewer, sorted; noise rows keep two links into two of the blobs, as a search that
    passed through them leaves behind.  [n, k] int32."""
    n = X.shape[0]
    out = torch.empty((n, k), dtype=torch.int64, device="cuda")
    blobs = _blobs(n)
    order = torch.argsort(which, stable=True)
    sizes = torch.bincount(which + 1, minlength=blobs + 1).tolist()
    first = np.cumsum([0] + sizes).tolist()
    for b in range(blobs + 1):
        rows = order[first[b]:first[b + 1]]
        parts = max(1, math.ceil(rows.numel() / 8192))
        for part in rows.chunk(parts):
            P = X[part]
            own = torch.arange(part.numel(), device="cuda")
            out[part] = part[_nearest(P, P, k, own)[1]]
            if b > 0 and part[0] != rows[0]:  # a blob's parts hang together through one link each
                out[part[0], k - 1] = rows[0]
    noise = order[:sizes[0]]
    j = torch.arange(noise.numel(), device="cuda")
    start = torch.tensor(first[1:-1], device="cuda")
    size = torch.tensor(sizes[1:], device="cuda")
    for back in (1, 2):
        b = (j + back) % blobs
        out[noise, k - back] = order[start[b] + (7 * j) % size[b]]
    return out.to(torch.int32)


def _pairs(X, ids):
    """The distance of every listed neighbour, in 64 bits."""
    out = torch.empty(ids.shape, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 27) // (ids.shape[1] * X.shape[1]))
    for a in range(0, ids.shape[0], step):
        i = ids[a:a + step].long()
        out[a:a + step] = (X[a:a + step, None, :].double() - X[i].double()).square().sum(2).sqrt()
    return out


def _instances(case):
    """The (n, d) of a batch's instances: sizes spread over the logarithm of their range."""
    r = random.Random(case["count"])
    dims = [int(x) for x in case["dims"].split(",")]
    return [(_log(r, case["n_lo"], case["n_hi"]), r.choice(dims)) for _ in range(case["count"])]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "ctx": _context()}
    if kind == "batch":
        s["X"] = [_points(n, d, seed * 1009 + i)[0] for i, (n, d) in enumerate(_instances(case))]
        return s
    if kind == "merge":  # two shards of one data set, each with its own graph
        P, _ = _points(case["n"] + case["n2"], case["d"], seed)
        s["X"], s["Y"] = P[:case["n"]].clone(), P[case["n"]:].clone()
        for name in ("X", "Y"):
            P = s[name]
            v, i = _nearest(P, P, case["k"], torch.arange(P.shape[0], device="cuda"))
            s["G" + name] = torch.stack([v.view(torch.int32), i.to(torch.int32)], dim=2).contiguous()
        return s
    X, which = _points(case["n"], case["d"], seed)
    s["X"] = X
    if kind == "run" and case["host"]:
        s["X"] = X.cpu()
    if kind in ("tail", "stages"):
        s["ids"] = _knn(X, which, case["k"])
        if kind == "tail":  # the graph as NNDescent hands it on: (distance bits, id) rows
            ids = s.pop("ids")
            dist = _pairs(X, ids).square().float()
            s["G"] = torch.stack([dist.view(torch.int32), ids], dim=2).contiguous()
    return s


# ---- one pass ------------------------------------------------------------------
def _euclidean(G):
    """The neighbour distances of a graph's rows ((squared distance bits, id) pairs)."""
    return G.view(torch.float32)[..., 0].sqrt()


def _room(t, rows):
    """An output whose length depends on the data, in an array of the length it has room for."""
    out = t.new_zeros((rows, *t.shape[1:]))
    out[:t.shape[0]] = t
    return out


def run(s):
    case, ctx, X = s["case"], s["ctx"], s["X"]
    kind, k = case["kind"], case["k"]
    if kind == "knn":
        G = ctx.NNDescent(X, k=k, sample_num=k // 2, iterations=_ITERATIONS,
                          precision=_PRECISION[case["precision"]])
        return _euclidean(G)
    if kind == "run":
        _, _, G = ctx.hdbscan(X, k=k, mpts=k, sample_num=k // 2, iterations=_ITERATIONS,
                              precision=_PRECISION[case["precision"]], want_graph=True)
        return _euclidean(G)
    if kind == "batch":
        _, _, _, graphs = ctx.hdbscan_batched(X, k=k, mpts=k, sample_num=k // 2,
                                              iterations=_ITERATIONS,
                                              precision=_PRECISION[case["precision"]],
                                              want_graphs=True, strict=False)
        return _euclidean(torch.cat(graphs))
    if kind == "tail":
        labels, stats = ctx.hdbscan_from_knn(s["G"], X, k=k, mpts=case["mpts"])
        return {"labels": labels, "edges": stats["edges"], "clusters": stats["num_clusters"]}
    if kind == "merge":
        G = ctx.KNNMerge(X, s["GX"], s["Y"], s["GY"], sample_num=_MERGE_SAMPLES,
                         iterations=_MERGE_ITERATIONS)
        return _euclidean(G)
    n = case["n"]
    ids = s["ids"]
    dist = ctx.fix_distances(X, ids)
    graph = ctx.buildEnhancedKNNG(ids, dist, X)
    mst, in_mst, _ = ctx.buildMST(graph, with_in_mst=True)
    by_ids, _, _ = ctx.buildMST(graph, order=hdb.HDB_ORDER_IDS)
    quantised, _, _, _ = ctx.buildMST_quantised(graph, dist)
    quantised = ctx.sort_edges(quantised)
    tree = ctx.build_Linkage_tree(mst, n)
    labels, clusters, condensed, stability = ctx.get_clusters(
        tree, n, case["mpts"], stability=hdb.HDB_STAB_FP64, want_tree=True)
    core_sg = ctx.build_CoreSG(ids, dist, X, mst)
    edges = 2 * n * k + math.isqrt(n) ** 2  # room for the most edges and rows that n and k allow
    rows = n + 2 * (n // case["mpts"]) + 2
    return {"dist": dist, "nindex": graph.nindex, "nlist": _room(graph.nlist, edges),
            "eweight": _room(graph.eweight, edges), "antihubs": graph.antihubs, "mst": mst,
            "in_mst": _room(in_mst, edges), "by_ids": by_ids, "quantised": quantised, "tree": tree,
            "labels": labels, "clusters": clusters, "condensed": _room(condensed, rows),
            "stability": _room(stability, rows), "sg_nindex": core_sg.nindex,
            "sg_nlist": _room(core_sg.nlist, edges + 2 * n),
            "sg_eweight": _room(core_sg.eweight, edges + 2 * n)}


# ---- what a pass cannot do without ------------------------------------------------
def _descent(n, d, k, iterations, samples, cross=False):
    """X read, the graph written; the sampled pairs' distances (3 operations a coordinate)."""
    pairs = samples * 2 * samples if cross else samples * (4 * samples - 1) // 2
    return 4 * n * d + 8 * n * k, 3.0 * d * n * pairs * iterations


def work(case):
    kind, k = case["kind"], case["k"]
    if kind == "batch":
        parts = [_descent(n, d, k, _ITERATIONS, k // 2) for n, d in _instances(case)]
        return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}
    n, d = case["n"], case["d"]
    if kind in ("knn", "run"):
        b, f = _descent(n, d, k, _ITERATIONS, k // 2)
        return {"bytes": b + (4 * n if kind == "run" else 0), "flops": f}
    if kind == "merge":
        m = n + case["n2"]
        b, f = _descent(m, d, k, _MERGE_ITERATIONS, _MERGE_SAMPLES, cross=True)
        return {"bytes": b + 8 * m * k, "flops": f}
    # graph stages: ids, X and about 1.5 k edges a row (id and weight) written once
    graph = 4 * n * k + 4 * n * d + 12 * n * k
    if kind == "tail":
        return {"bytes": graph + 4 * n * k + 4 * n, "flops": 3.0 * n * d}
    # + distances, three MSTs, the trees, and Core-SG's edges
    return {"bytes": graph + 4 * n * k + n * (3 * 12 + 16 + 16 + 8) + 12 * n * k,
            "flops": 3.0 * n * k * d}


# ---- the same in 64 bits -----------------------------------------------------------
def _exact_knn(X, k):
    """Every row's true neighbour distances, which the graphs approach."""
    X = X.cuda().double()
    return _nearest(X, X, k, torch.arange(X.shape[0], device="cuda"))[0].sqrt()


def exact(case, seed):
    kind = case["kind"]
    if kind == "stages":
        s = prepare(case, seed)
        return {"dist": _pairs(s["X"], s["ids"])}
    if kind == "batch":
        if max(n for n, _ in _instances(case)) > 100_000:
            return None
        return torch.cat([_exact_knn(X, case["k"]) for X in prepare(case, seed)["X"]])
    points = case.get("n", 0) + case.get("n2", 0)
    if kind == "tail" or points > 200_000:  # labels are whole numbers; larger graphs take too long
        return None
    if kind == "merge":
        s = prepare(case, seed)
        return _exact_knn(torch.cat([s["X"], s["Y"]]), case["k"])
    return _exact_knn(_points(case["n"], case["d"], seed)[0], case["k"])
