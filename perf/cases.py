"""The work that programs built on this package do, as measurable cases.

Each case is one pass through the package's public entry points on a graph of
its own: traversals (top-down, direction-optimising, many graphs at once),
triangle counts, connected components, k-truss, dynamic updates and a mix of
all of them as a server runs it.  Every output is integer, so outputs are
compared exactly.
"""
import math

import numpy as np
import torch

import hornet_b200 as H
from hornet_b200.batching import GraphBatch, synthetic_specs

DEV = "cuda:0"


def listed():
    return [
        # one traversal request on a small graph: launches and latency
        {"name": "bfs_small", "path": "bfs", "graph": "rmat", "nV": 1 << 12, "ef": 16, "k": 1},
        # the benchmark's traversal: 16 sources of the scale-22 graph, distances kept on the device
        {"name": "bfs_topdown", "path": "bfs", "graph": "rmat", "nV": 1 << 22, "ef": 16, "k": 16},
        # the same sources through the direction-optimising traversal
        {"name": "bfs_diropt", "path": "bfs_do", "graph": "rmat", "nV": 1 << 22, "ef": 16, "k": 16},
        # a road-like network: hundreds of levels of small frontiers
        {"name": "bfs_road", "path": "bfs", "graph": "grid", "nV": 240999, "ef": 2, "k": 1},
        # many small graphs of uneven size held as one: 8 traversals and a triangle count of each
        {"name": "batch_graphs", "path": "batch", "graphs": 512, "k": 8},
        # triangles of the benchmark graph
        {"name": "tc_large", "path": "tc", "graph": "rmat", "nV": 1 << 22, "ef": 16},
        # components of the benchmark graph
        {"name": "cc_large", "path": "cc", "graph": "rmat", "nV": 1 << 22, "ef": 16},
        # truss numbers of all edges of a mid-size graph of odd size
        {"name": "ktruss", "path": "ktruss", "graph": "rmat", "nV": 100003, "ef": 16},
        # a small batch that arrives in host memory: inserted, the graph read out, erased again
        {"name": "update_small", "path": "update", "graph": "rmat", "nV": 1 << 18, "ef": 16,
         "batch": 1000, "pairs": "uniform", "dedup": True, "host": True},
        # an ordinary batch with the graph's own skew (hubs, duplicates), odd sizes
        {"name": "update_skewed", "path": "update", "graph": "rmat", "nV": 3000017, "ef": 12,
         "batch": 300007, "pairs": "rmat", "dedup": True, "host": False},
        # the largest batch
        {"name": "update_large", "path": "update", "graph": "rmat", "nV": 1 << 23, "ef": 16,
         "batch": 10000000, "pairs": "uniform", "dedup": True, "host": False},
        # a serving step: a coalesced run of updates, a traversal, local triangle counts, the run undone
        {"name": "serve_step", "path": "serve", "graph": "rmat", "nV": 1 << 21, "ef": 16,
         "batch": 20000, "seeds": 1000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["bfs", "bfs", "bfs_do", "batch", "tc", "cc", "ktruss", "update", "update",
                       "serve"])
    if path == "batch":
        return {"path": path, "graphs": _log(rng, 8, 512), "k": rng.randint(1, 8)}
    c = {"path": path, "graph": rng.choice(["rmat", "rmat", "uniform"])}
    hi = {"ktruss": 100003, "serve": 1 << 21, "update": 1 << 22}.get(path, 1 << 22)
    if path == "bfs" and rng.random() < 0.25:
        c.update(graph="grid", nV=_log(rng, 5000, 240999), ef=2, k=rng.randint(1, 2))
        return c
    c["nV"] = _log(rng, 1 << 12, hi)
    c["ef"] = rng.randint(4, 16)
    if path in ("bfs", "bfs_do"):
        c["k"] = rng.randint(1, 16)
    elif path == "update":
        c["batch"] = _log(rng, 500, min(3000000, c["nV"] * c["ef"] // 4))
        c["pairs"] = rng.choice(["uniform", "rmat"])
        c["dedup"] = rng.random() < 0.75
        c["host"] = rng.random() < 0.25 and c["batch"] < 100000
    elif path == "serve":
        c["batch"] = _log(rng, 100, min(100000, c["nV"]))
        c["seeds"] = rng.randint(1, min(1000, c["nV"]))
    return c


def _pairs(kind, nV, count, seed):
    """`count` vertex pairs on the device: R-MAT or uniform over [0, nV)."""
    src = torch.empty(count, dtype=torch.int32, device=DEV)
    dst = torch.empty_like(src)
    abc = {} if kind == "rmat" else {"a": 0.25, "b": 0.25, "c": 0.25}
    H.gen_rmat_device(max(1, (nV - 1).bit_length()), count, seed, src, dst, n_vertices=nV, **abc)
    return src, dst


def _grid_pairs(nV, seed):
    """Street-like pairs: a lattice about 1.5 times as wide as high, every tenth link missing."""
    w = int(math.sqrt(1.5 * nV))
    g = torch.Generator(device=DEV).manual_seed(seed)
    v = torch.arange(nV, device=DEV)
    right = v[(v % w != w - 1) & (v + 1 < nV)]
    down = v[v + w < nV]
    src = torch.cat([right, down])
    dst = torch.cat([right + 1, down + w])
    keep = torch.rand(len(src), generator=g, device=DEV) > 0.1
    return src[keep].to(torch.int32), dst[keep].to(torch.int32)


def _trim(nV, src, dst, count, seed):
    """`count` of the distinct pairs, so that graphs of all seeds have as many edges."""
    s, d = src.to(torch.int64), dst.to(torch.int64)
    key = torch.unique((torch.minimum(s, d) * nV + torch.maximum(s, d))[s != d])
    g = torch.Generator(device=DEV).manual_seed(seed)
    key = key[torch.randperm(len(key), generator=g, device=DEV)[:count]]
    return (key // nV).to(torch.int32), (key % nV).to(torch.int32)


def _union(case, seed):
    """Graphs of uneven size (the sizes and kinds of batching.synthetic_specs,
    the same for every seed; the edges from the seed) as one graph."""
    sizes, bases, _, specs = synthetic_specs(case["graphs"])
    ends = np.cumsum([sp[1] for sp in specs])
    src = torch.empty(int(ends[-1]), dtype=torch.int32, device=DEV)
    dst = torch.empty_like(src)
    for i, (scale, count, _, n, a, b, c) in enumerate(specs):
        s, d = src[ends[i] - count:ends[i]], dst[ends[i] - count:ends[i]]
        H.gen_rmat_device(scale, count, seed * 1_000_003 + i, s, d, n_vertices=n, a=a, b=b, c=c)
        s += int(bases[i])
        d += int(bases[i])
    torch.cuda.synchronize()
    h = H.hornet_from_device_csr(H.coo_to_csr_device(int(sizes.sum()), src, dst))
    return h, sizes, bases


def _graph(case, seed):
    """An undirected graph without loops and duplicates, and the pairs it was made of."""
    nV = case["nV"]
    if case["graph"] == "grid":
        src, dst = _grid_pairs(nV, seed)
    else:
        src, dst = _pairs(case["graph"], nV, nV * case["ef"], seed)
    if case["path"] == "ktruss":
        src, dst = _trim(nV, src, dst, int(0.7 * nV * case["ef"]), seed)
    torch.cuda.synchronize()
    return H.hornet_from_device_csr(H.coo_to_csr_device(nV, src, dst)), src, dst


def _sources(src, dst, k, rng):
    """k vertices that have an edge."""
    at = torch.from_numpy(rng.integers(0, len(src), 64 * k)).to(src.device)
    s, d = src[at].cpu().numpy(), dst[at].cpu().numpy()
    return np.ascontiguousarray(s[s != d][:k])


def prepare(case, seed):
    path = case["path"]
    rng = np.random.default_rng(seed)
    if path == "batch":
        h, sizes, bases = _union(case, seed)
        b = GraphBatch(h, bases, sizes)
        src = (rng.random((len(sizes), case["k"])) * sizes[:, None]).astype(np.int64)
        return {"case": case, "h": h, "b": b, "src": src,
                "dist": torch.empty((case["k"], h.nV()), dtype=torch.int32, device=DEV),
                "pv": torch.empty(h.nV(), dtype=torch.int64, device=DEV)}
    h, src, dst = _graph(case, seed)
    s = {"case": case, "h": h}
    nV = case["nV"]
    if path in ("bfs", "bfs_do"):
        s["alg"] = H.BfsTopDown(h)
        s["sources"] = _sources(src, dst, case["k"], rng)
        s["out"] = torch.empty((len(s["sources"]), nV), dtype=torch.int32, device=DEV)
    elif path == "tc":
        s["alg"] = H.TriangleCounting2(h)
    elif path == "cc":
        s["alg"] = H.CC(h)
        s["out"] = torch.empty(nV, dtype=torch.int32, device=DEV)
    elif path == "ktruss":
        s["alg"] = H.KTruss(h)
    elif path == "update":
        bs, bd = _pairs(case["pairs"], nV, case["batch"], seed + 1)
        s["batch"] = (bs.cpu().numpy(), bd.cpu().numpy()) if case["host"] else (bs, bd)
        # room for any graph of this case's pairs with the batch in it
        room = 2 * nV * case["ef"] + case["batch"]
        s["coo"] = (torch.full((room,), -1, dtype=torch.int32, device=DEV),
                    torch.full((room,), -1, dtype=torch.int32, device=DEV))
    elif path == "serve":
        # new pairs to insert and existing ones to erase, both directions of each
        n = case["batch"]
        i_s, i_d = (t.cpu().numpy() for t in _pairs("rmat", nV, n, seed + 1))
        at = torch.from_numpy(rng.integers(0, len(src), n)).to(src.device)
        e_s, e_d = src[at].cpu().numpy(), dst[at].cpu().numpy()
        ins = (np.concatenate([i_s, i_d]), np.concatenate([i_d, i_s]))
        era = (np.concatenate([e_s, e_d]), np.concatenate([e_d, e_s]))
        ops = np.repeat(np.array([1, 0], np.uint8), [2 * n, 2 * n])
        s["do"] = (np.concatenate([ins[0], era[0]]), np.concatenate([ins[1], era[1]]), ops)
        s["undo"] = (np.concatenate([era[0], ins[0]]), np.concatenate([era[1], ins[1]]), ops)
        s["bfs"] = H.BfsTopDown(h)
        s["sources"] = _sources(src, dst, 1, rng)
        s["out"] = torch.empty((1, nV), dtype=torch.int32, device=DEV)
        s["tc"] = H.TriangleCounting2(h)
        s["seeds"] = torch.from_numpy(rng.integers(0, nV, case["seeds"]).astype(np.int32)).to(DEV)
        s["local"] = torch.empty(case["seeds"], dtype=torch.int64, device=DEV)
    return s


def run(s):
    path, h = s["case"]["path"], s["h"]
    if path == "batch":
        s["b"].bfs(s["src"], s["dist"])
        per_graph, total = s["b"].triangles(s["pv"])
        return s["dist"], s["pv"], per_graph, total
    if path in ("bfs", "bfs_do"):
        out, stats = s["alg"].run_multi(s["sources"], out=s["out"],
                                        direction_optimizing=path == "bfs_do")
        return out, [x.levels for x in stats], [x.visited for x in stats]
    if path == "tc":
        return s["alg"].run()
    if path == "cc":
        return s["alg"].run(out=s["out"]), s["alg"].n_components
    if path == "ktruss":
        return s["alg"].run(), s["alg"].edge_truss
    if path == "update":
        dedup = s["case"]["dedup"]
        b = H.BatchUpdate(h, *s["batch"])
        added = h.insert(b, removeBatchDuplicates=dedup, removeGraphDuplicates=dedup)
        coo = h.getCOO(True, *s["coo"])
        removed = h.erase(b, removeBatchDuplicates=dedup)
        return added, coo, removed, h.nE()
    done = h.update_coalesced(*s["do"])
    out, stats = s["bfs"].run_multi(s["sources"], out=s["out"], direction_optimizing=True)
    s["tc"].local(s["seeds"], out=s["local"])
    undone = h.update_coalesced(*s["undo"])
    return done, out, stats[0].levels, s["local"], undone


def _size(case):
    """(vertices, directed edges) of a case's graph, the edges from the mean
    share of pairs that are no loops or repeats."""
    if case["path"] == "batch":
        # sizes are log-uniform in [1024, 65536]; half the graphs have 4 pairs a vertex, half 16
        n = case["graphs"] * 64512 / math.log(64)
        return n, 2 * n * (4 + 16 * 0.84) / 2
    n, ef = case["nV"], case["ef"]
    if case["graph"] == "grid":
        return n, 3.6 * n
    if case["path"] == "ktruss":
        return n, 2 * int(0.7 * n * ef)
    keep = 1.0 if case["graph"] == "uniform" else min(0.97, 0.72 + 0.0235 * (math.log2(n) - 12))
    return n, 2 * n * ef * keep


def work(case):
    """Bytes that a pass cannot do without: the adjacency (4 an edge) and the
    row bounds (8 a vertex) read once, the results written once."""
    path = case["path"]
    n, m = _size(case)
    graph = 4 * m + 8 * n
    if path in ("bfs", "bfs_do"):
        b = case["k"] * (graph + 4 * n)
    elif path == "batch":
        b = case["k"] * 4 * n + graph + graph + 8 * n
    elif path == "tc":
        b = graph + 8
    elif path == "cc":
        b = graph + 4 * n
    elif path == "ktruss":
        b = graph + 4 * m
    elif path == "update":
        # the batch read and its edges written and taken out, the graph read and written out
        b = 2 * (8 + 4) * case["batch"] + graph + 8 * m
    else:
        b = 2 * (9 + 4) * 4 * case["batch"] + graph + 4 * n + 12 * case["seeds"]
    return {"bytes": float(b), "flops": 0.0}


def tolerance(case):
    return "exact"
