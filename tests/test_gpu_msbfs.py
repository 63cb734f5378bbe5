"""GPU parity of the batched BFS (hn_bfs_batch): up to 64 BFS slots in one
traversal.  Every slot's distances are compared bit-exactly with the
oracle's single-source BFS (the restatement of
hornetsnest/src/Static/BreadthFirstSearch/TopDown.cu), and the per-slot
statistics with the oracle's counts."""
import numpy as np
import pytest

import hornet_b200 as H
from oracle import oracle as O
from tests import helpers as T

pytestmark = pytest.mark.gpu


def build(g: O.Csr) -> H.Hornet:
    return H.Hornet(H.HornetInit(g.nV, g.nE, g.off32(), g.adj, sorted_adjacency=True))


def oracle_slots(g, sources, slots, nslots):
    """Per slot: the minimum over its sources of the single-source BFS
    distance (the multi-source BFS distance), with visited/scanned/levels."""
    dist = np.full((nslots, g.nV), O.INF, np.int64)
    for s, b in zip(sources, slots):
        d, _ = O.bfs(g, int(s))
        dist[b] = np.minimum(dist[b], d)
    stats = []
    for b in range(nslots):
        reached = dist[b] != O.INF
        deg = np.diff(g.off)
        lv = int(dist[b][reached].max()) + 1 if reached.any() else 0
        stats.append((int(reached.sum()), int(deg[reached].sum()), lv))
    return dist.astype(np.int32), stats


def check(out, st, ref, ref_stats):
    np.testing.assert_array_equal(out, ref)
    for b, (vis, scanned, lv) in enumerate(ref_stats):
        assert st[b].visited == vis, b
        assert st[b].edges_scanned == scanned, b
        assert st[b].levels == lv, b


@pytest.mark.parametrize("name,k", [("rmat10", 64), ("er2000", 17), ("rmat12_nonpow2", 64)])
def test_batch_one_source_per_slot(name, k):
    g = {"rmat10": lambda: T.rmat_graph(10, 16, seed=3),
         "er2000": lambda: T.er_graph(2000, 8, seed=5),
         "rmat12_nonpow2": lambda: T.rmat_graph(12, 8, seed=7, n_vertices=3000)}[name]()
    h = build(g)
    rng = np.random.default_rng(11)
    srcs = np.concatenate([[0], rng.integers(0, g.nV, k - 1)]).astype(np.int32)
    out, st = H.BfsTopDown(h).run_batch(srcs)
    ref, ref_stats = oracle_slots(g, srcs, range(k), k)
    check(out, st, ref, ref_stats)
    # the same as k single-source runs through hn_bfs_multi
    multi, mst = H.BfsTopDown(h).run_multi(srcs)
    np.testing.assert_array_equal(out, multi)
    for b in range(k):
        assert st[b].levels == mst[b].levels


def test_batch_duplicate_sources_and_sparse_slots():
    g = T.rmat_graph(11, 8, seed=9)
    h = build(g)
    # the same vertex in several slots, two sources in one slot, slots 3..7 empty
    srcs = np.array([5, 5, 17, 900, 5, 5], np.int32)
    slots = np.array([0, 1, 1, 2, 8, 8], np.int32)
    out, st = H.BfsTopDown(h).run_batch(srcs, slots=slots, nslots=9)
    ref, ref_stats = oracle_slots(g, srcs, slots, 9)
    check(out, st, ref, ref_stats)
    assert (out[3:8] == O.INF).all()


def test_batch_disjoint_union_many_graphs():
    """4096-graph pattern, scaled down: 96 small graphs in one union, one
    source per graph, 8 slots; every graph's distances equal its own BFS."""
    graphs = [T.rmat_graph(6, 4, seed=100 + i) if i % 3 else T.er_graph(50, 3, seed=i)
              for i in range(96)]
    u, base = T.disjoint_union(graphs)
    h = build(u)
    rng = np.random.default_rng(3)
    srcs = np.array([base[i] + rng.integers(0, graphs[i].nV) for i in range(96)], np.int32)
    slots = np.arange(96, dtype=np.int32) % 8
    out, st = H.BfsTopDown(h).run_batch(srcs, slots=slots, nslots=8)
    for i, gi in enumerate(graphs):
        d, _ = O.bfs(gi, int(srcs[i] - base[i]))
        np.testing.assert_array_equal(out[slots[i], base[i]:base[i] + gi.nV], d)
    ref, ref_stats = oracle_slots(u, srcs, slots, 8)
    check(out, st, ref, ref_stats)


def test_batch_after_updates_and_isolated():
    g = T.rmat_graph(10, 8, seed=21)
    h = build(g)
    bfs = H.BfsTopDown(h)
    srcs = np.arange(0, 640, 10, dtype=np.int32)
    out0, _ = bfs.run_batch(srcs)
    np.testing.assert_array_equal(out0, oracle_slots(g, srcs, range(64), 64)[0])
    s, d = T.uniform_new_edges(g, 3000, seed=2)
    h.insert(H.BatchUpdate(h, s, d), removeBatchDuplicates=True, removeGraphDuplicates=True)
    g2, _ = O.insert(g, s, d, 3)
    out1, st1 = bfs.run_batch(srcs)
    ref, ref_stats = oracle_slots(g2, srcs, range(64), 64)
    check(out1, st1, ref, ref_stats)


def test_batch_device_output_and_errors():
    import torch
    g = T.er_graph(500, 4, seed=1)
    h = build(g)
    srcs = np.array([1, 2, 3], np.int32)
    dev = torch.empty((3, g.nV), dtype=torch.int32, device="cuda")
    H.BfsTopDown(h).run_batch(srcs, out=dev)
    np.testing.assert_array_equal(dev.cpu().numpy(), oracle_slots(g, srcs, range(3), 3)[0])
    with pytest.raises(H.HornetError):
        H.BfsTopDown(h).run_batch(np.arange(65, dtype=np.int32) % g.nV, nslots=65)
    with pytest.raises(H.HornetError):
        H.BfsTopDown(h).run_batch(srcs, slots=np.array([0, 1, 4], np.int32), nslots=4 - 1)
    with pytest.raises(H.HornetError):
        H.BfsTopDown(h).run_batch(np.array([g.nV], np.int32))


@pytest.mark.parametrize("block,ctas,bu", [(128, 2, 1), (512, 8, 0), (256, 6, 1), (256, 4, 0)])
def test_batch_block_size_knobs(block, ctas, bu):
    """Every batched-BFS launch shape the autotuner may pick gives the same
    distances (the CUDA graph is rebuilt when a knob changes)."""
    g = T.rmat_graph(11, 16, seed=13)
    h = build(g)
    srcs = np.arange(0, 2048, 64, dtype=np.int32)
    ref, ref_stats = oracle_slots(g, srcs, range(len(srcs)), len(srcs))
    try:
        H.tune_set("msbfs.block", block)
        H.tune_set("msbfs.ctas_per_sm", ctas)
        H.tune_set("msbfs.bottom_up", bu)
        H.tune_set("msbfs.check_min", 1)
        out, st = H.BfsTopDown(h).run_batch(srcs)
        check(out, st, ref, ref_stats)
    finally:
        H.tune_reset()


@pytest.mark.parametrize("alpha,beta", [(1, 1 << 20), (1 << 20, 1), (14, 24), (1 << 20, 1 << 20)])
def test_batch_bottom_up_switching(alpha, beta):
    """Bottom-up levels for the largest frontiers only (alpha 1), never (beta
    1: no frontier holds all vertices), from alpha 14 and beta 24, and from the
    first level on (both huge): distances and statistics unchanged."""
    g = T.rmat_graph(12, 16, seed=23)
    h = build(g)
    srcs = np.arange(0, 4096, 97, dtype=np.int32)
    ref, ref_stats = oracle_slots(g, srcs, range(len(srcs)), len(srcs))
    try:
        H.tune_set("msbfs.bottom_up", 1)
        H.tune_set("msbfs.check_min", 1)
        H.tune_set("bfs.do_alpha", alpha)
        H.tune_set("bfs.do_beta", beta)
        out, st = H.BfsTopDown(h).run_batch(srcs)
        check(out, st, ref, ref_stats)
    finally:
        H.tune_reset()


@pytest.mark.parametrize("block", [128, 256, 512])
def test_batch_bottom_up_long_lists(block):
    """Bottom-up levels over lists that a lane leaves to its warp (more than
    16 neighbours, up to a hub of 5,000), lists of capacity 1, 2 and 4, and
    vertices that some slots never reach."""
    rng = np.random.default_rng(2)
    star = O.build_csr_undirected(5001, np.zeros(5000, np.int32), np.arange(1, 5001, dtype=np.int32))
    path = O.build_csr_undirected(9, np.arange(8, dtype=np.int32), np.arange(1, 9, dtype=np.int32))
    g, base = T.disjoint_union([star, T.rmat_graph(11, 16, seed=3), path, T.er_graph(500, 60, seed=1)])
    h = build(g)
    srcs = np.concatenate([base, rng.integers(0, g.nV, 36), [5000, int(base[2]) + 8]]).astype(np.int32)
    slots = np.arange(len(srcs)) % 40
    ref, ref_stats = oracle_slots(g, srcs, slots, 40)
    try:
        H.tune_set("msbfs.block", block)
        H.tune_set("msbfs.check_min", 1)
        for alpha, beta in ((1 << 20, 1), (1 << 20, 1 << 20), (2, 24)):
            H.tune_set("bfs.do_alpha", alpha)
            H.tune_set("bfs.do_beta", beta)
            out, st = H.BfsTopDown(h).run_batch(srcs, slots=slots.astype(np.int32), nslots=40)
            check(out, st, ref, ref_stats)
    finally:
        H.tune_reset()


@pytest.mark.parametrize("extra", [-1, 0, 1, 700])
@pytest.mark.parametrize("slots", [1, 9])
def test_batch_levels_without_a_touched_list(extra, slots):
    """Frontiers of about nV / 4 edges: one more and the level records no
    list of touched vertices.  Two hubs share leaves, which lead on to more
    vertices; some slots start at a leaf or an isolated vertex."""
    n = 4000
    d = n // 4 + extra - 1
    leaves = np.arange(2, 2 + d)
    s = np.concatenate([np.zeros(d), [0], np.ones(d // 2), leaves[: d // 3]]).astype(np.int32)
    t = np.concatenate([leaves, [1], leaves[: d // 2], leaves[: d // 3] + d]).astype(np.int32)
    g = O.build_csr_undirected(n, s, t)
    h = build(g)
    srcs = np.array([0, 2, n - 1, 1, d, 2 + d, 0, 5, 9][:slots], np.int32)
    ref, ref_stats = oracle_slots(g, srcs, range(slots), slots)
    try:
        H.tune_set("msbfs.check_min", 1)
        for bu in (0, 1):
            H.tune_set("msbfs.bottom_up", bu)
            out, st = H.BfsTopDown(h).run_batch(srcs)
            check(out, st, ref, ref_stats)
    finally:
        H.tune_reset()


def one_way_layers(width, layers):
    """Vertex 0, then layers of `width` vertices with four edges each to the
    next layer; the last layer has no edges.  Nothing leads back."""
    n = 1 + width * layers
    at = 1 + width * np.arange(layers)
    i = np.arange(width)
    src, dst = [np.zeros(width, np.int64)], [at[0] + i]
    for a, b in zip(at[:-1], at[1:]):
        for step in (0, 1, 3, 7):
            src.append(a + i)
            dst.append(b + (i + step) % width)
    return one_way(n, np.concatenate(src), np.concatenate(dst))


def one_way(n, src, dst):
    order = np.lexsort((dst, src))
    off = np.zeros(n + 1, np.int64)
    np.add.at(off, src + 1, 1)
    return O.Csr(np.cumsum(off), dst[order].astype(np.int32))


@pytest.mark.parametrize("width,layers", [(30, 20), (1000, 20), (1000, 3)])
@pytest.mark.parametrize("slots", [1, 9])
def test_batch_one_way_graph(width, layers, slots):
    """Edges stored one way only: no level may look for predecessors in a
    vertex's own list, whichever directions are allowed."""
    g = one_way_layers(width, layers)
    h = build(g)
    srcs = (np.arange(slots) * 7 % (1 + width)).astype(np.int32)
    ref, ref_stats = oracle_slots(g, srcs, range(slots), slots)
    try:
        for alpha, beta in ((4, 24), (14, 24), (1 << 20, 1 << 20)):
            H.tune_set("bfs.do_alpha", alpha)
            H.tune_set("bfs.do_beta", beta)
            for _ in range(2):
                out, st = H.BfsTopDown(h).run_batch(srcs)
                check(out, st, ref, ref_stats)
    finally:
        H.tune_reset()


def test_batch_graph_loses_and_regains_an_edge():
    """A symmetric graph, the same after updates that store the only edge to
    a vertex one way, and after one that stores it both ways again."""
    core = T.rmat_graph(11, 16, seed=17)
    n = core.nV + 1
    s, d = core.coo()
    hub = int(np.diff(core.off).argmax())
    g = one_way(n, np.concatenate([s, [hub, n - 1]]), np.concatenate([d, [n - 1, hub]]))
    h = build(g)
    srcs = np.concatenate([[hub], np.arange(0, 2000, 61)]).astype(np.int32)

    def same():
        ref, ref_stats = oracle_slots(g, srcs, range(len(srcs)), len(srcs))
        out, st = H.BfsTopDown(h).run_batch(srcs)
        check(out, st, ref, ref_stats)

    try:
        H.tune_set("bfs.do_alpha", 1 << 20)
        H.tune_set("bfs.do_beta", 1 << 20)
        same()
        back = np.array([n - 1], np.int32), np.array([hub], np.int32)
        assert h.erase(H.BatchUpdate(h, *back)) == 1
        g, _ = O.erase(g, *back, 0)
        same()
        assert h.insert(H.BatchUpdate(h, *back), True, True) == 1
        g, _ = O.insert(g, *back, 3)
        same()
    finally:
        H.tune_reset()


@pytest.mark.parametrize("run", [lambda: test_batch_bottom_up_switching(1 << 20, 1 << 20),
                                 lambda: test_batch_bottom_up_long_lists(256),
                                 lambda: test_batch_one_way_graph(1000, 3, 9),
                                 test_batch_graph_loses_and_regains_an_edge])
def test_batch_small_graphs_checked_for_one_way_edges(run):
    """The check for edges stored one way, and the pulls after it, on graphs
    below the size from which it is made by default."""
    H.tune_set("msbfs.check_min", 1)
    H.profile_enable(True)
    try:
        run()
        assert "k_ms_one_way" in H.profile_report()
    finally:
        H.profile_enable(False)
        H.tune_reset()
