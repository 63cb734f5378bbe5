"""The one-launch BFS where a level changes hands: frontiers at the limit of
CTA 0's small levels, thin grid-wide levels, small levels that reach hubs
(chunk marks left to the grid), bottom-up levels with hubs off the frontier,
and switches between the directions.  Distances and statistics equal the
oracle's, for every grid size and with one launch per level."""
import numpy as np
import pytest

import hornet_b200 as H
from oracle import oracle as O
from tests import helpers as T

pytestmark = pytest.mark.gpu


def build(g):
    return H.Hornet(H.HornetInit(g.nV, g.nE, g.off32(), g.adj, sorted_adjacency=True))


def two_level_star(first, leaves):
    """Source 0 - `first` neighbours, neighbour i with leaves[i] leaves."""
    leaves = np.asarray(leaves, np.int64)
    s = [np.zeros(first, np.int64), np.repeat(1 + np.arange(first), leaves)]
    d = [1 + np.arange(first), 1 + first + np.arange(leaves.sum())]
    n = 1 + first + int(leaves.sum())
    return O.build_csr_undirected(n, np.concatenate(s).astype(np.int32),
                                  np.concatenate(d).astype(np.int32))


def shape(kind):
    if kind.startswith("frontier_"):           # second level of exactly that many edges
        total = int(kind.split("_")[1])
        first = 1000
        leaves = np.full(first, (total - first) // first)
        leaves[0] += total - first - leaves.sum()
        return two_level_star(first, leaves)
    if kind == "hubs_from_small":              # 300 hubs reached by a level of 300 edges
        return two_level_star(300, np.full(300, 8000))
    if kind == "wide_star":                    # one hub over many chunks, then thin levels
        return two_level_star(150_000, np.repeat([1, 0], 75_000))
    if kind == "long_path":
        p = np.random.default_rng(3).permutation(3000).astype(np.int32)
        return O.build_csr_undirected(3000, p[:-1], p[1:])
    if kind == "dense":
        return T.er_graph(3000, 400, seed=9)
    return T.rmat_graph(15, 16, seed=21)


KINDS = ["frontier_4095", "frontier_4096", "frontier_4097", "frontier_120000", "hubs_from_small",
         "wide_star", "long_path", "dense", "rmat"]


@pytest.mark.parametrize("kind", KINDS)
def test_levels_change_hands(kind):
    g = shape(kind)
    h = build(g)
    srcs = [0, g.nV - 1, g.nV // 2]
    refs = [O.bfs(g, s) for s in srcs]
    settings = [{}, {"bfs.warp_ctas_per_sm": 1}, {"bfs.do_alpha": 1 << 20, "bfs.do_beta": 1},
                {"bfs.do_alpha": 2, "bfs.do_beta": 1 << 20}]
    if kind != "long_path":
        settings += [{"bfs.host_levels": 1, "bfs.do_alpha": 1 << 20},
                     {"bfs.host_levels": 1, "bfs.warp_ctas_per_sm": 2}]
    for knobs in settings:
        try:
            for k, v in knobs.items():
                H.tune_set(k, v)
            for do in (False, True):
                out, st = H.BfsTopDown(h).run_multi(srcs, direction_optimizing=do)
                for i in range(len(srcs)):
                    ref, scanned = refs[i]
                    np.testing.assert_array_equal(out[i], ref)
                    reached = ref != O.INF
                    assert st[i].edges_scanned == scanned
                    assert st[i].visited == int(reached.sum())
                    assert st[i].levels == int(ref[reached].max()) + 1
        finally:
            H.tune_reset()


def test_unaligned_distance_rows():
    """Rows of a multi-source call that do not start on 16 bytes."""
    import torch
    g = T.rmat_graph(12, 8, seed=5, n_vertices=3001)
    h = build(g)
    srcs = [3, 5, 9, 2999]
    buf = torch.full((4 * 3001 + 1,), -7, dtype=torch.int32, device="cuda:0")
    torch.cuda.synchronize()
    H.BfsTopDown(h).run_multi(srcs, out=buf[1:].view(4, 3001))
    out = buf.cpu().numpy()
    assert out[0] == -7
    for i, s in enumerate(srcs):
        np.testing.assert_array_equal(out[1 + i * 3001:1 + (i + 1) * 3001], O.bfs(g, s)[0])


@pytest.mark.parametrize("views", [2, 3, 8])
def test_views_share_the_gpu(views):
    """BFS calls on several views at once: launches of all grid sizes from the
    whole GPU to a share of it, also down to one CTA's levels."""
    import threading
    import torch
    g = shape("rmat")
    h = build(g)
    vs = [h.view() for _ in range(views)]
    srcs = [0, g.nV - 1, g.nV // 2, 5]
    refs = np.stack([O.bfs(g, s)[0] for s in srcs])
    wrong, start = [], threading.Barrier(views)

    def traverse(i):
        bfs = H.BfsTopDown(vs[i])
        out = torch.empty((len(srcs), g.nV), dtype=torch.int32, device="cuda:0")
        start.wait()
        for r in range(10):
            bfs.run_multi(srcs, out=out, direction_optimizing=(i + r) % 2 == 1)
            if not (out.cpu().numpy() == refs).all():
                wrong.append((i, r))

    threads = [threading.Thread(target=traverse, args=(i,)) for i in range(views)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
