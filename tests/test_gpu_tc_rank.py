"""Triangle counts by bitmaps: the rank orientation (graphs of more than 131,072
vertices whose edges are not local in id): totals, per-vertex and owner
counts equal the id orientation's (tc.flip = 0 never ranks) and the oracle's,
with lists inside, across and beyond the bitmaps (65,535 numbers for a
warp, 131,072 for a CTA)."""
import ctypes

import numpy as np
import pytest

import hornet_b200 as H
from oracle import oracle as O
from tests import helpers as T

pytestmark = pytest.mark.gpu


def build(g):
    return H.Hornet(H.HornetInit(g.nV, g.nE, g.off32(), g.adj, sorted_adjacency=True))


def owner(h):
    out = np.zeros(h.nV(), np.uint64)
    total = ctypes.c_uint64()
    H._check(H.lib().hn_tc_owner(h.handle, out.ctypes.data_as(ctypes.c_void_p), H.HN_MEM_HOST,
                                 ctypes.byref(total)))
    return out, total.value


def graph(kind):
    rng = np.random.default_rng(3)
    if kind == "rmat":
        return T.rmat_graph(18, 8, seed=2)
    if kind == "uniform":       # lists mostly beyond the windows
        return T.er_graph(200_001, 24, seed=4)
    if kind == "sparse_core":   # a dense core of scattered ids, lists across the window's edge
        n = 140_000
        core = rng.permutation(n)[:600].astype(np.int32)
        s = [core[rng.integers(0, 600, 240_000)], rng.integers(0, n, 300_000).astype(np.int32)]
        d = [core[rng.integers(0, 600, 240_000)], core[rng.integers(0, 600, 300_000)]]
        return O.build_csr_undirected(n, np.concatenate(s), np.concatenate(d))
    return O.build_csr_undirected(131_073, rng.integers(0, 131_073, 900_000).astype(np.int32),
                                  rng.integers(0, 131_073, 900_000).astype(np.int32))


@pytest.mark.parametrize("kind", ["rmat", "uniform", "sparse_core", "just_over"])
def test_rank_orientation(kind):
    g = graph(kind)
    h = build(g)
    ref = O.tc(g)
    tc = H.TriangleCounting2(h)
    for knobs in ({}, {"tc.warp_cap": 32, "tc.warp_work": 1024, "tc.mid_cap": 32,
                       "tc.item_work": 1024}):
        try:
            for k, v in knobs.items():
                H.tune_set(k, v)
            assert tc.run() == ref
            assert tc.run(per_vertex=True) == ref
            pv = tc.copyTCToHost().copy()
            ow, total = owner(h)
            H.tune_set("tc.flip", 0)
            assert total == ref == int(ow.sum())
            assert tc.run(per_vertex=True) == ref
            np.testing.assert_array_equal(pv, tc.copyTCToHost())
            ow0, _ = owner(h)
            np.testing.assert_array_equal(ow, ow0)
        finally:
            H.tune_reset()


def test_lists_too_long_for_the_table_go_by_id():
    """tc.cta_table_cap below the longest oriented list: no ranking."""
    g = T.rmat_graph(18, 8, seed=6, n_vertices=140_003)
    h = build(g)
    try:
        H.tune_set("tc.cta_table_cap", 64)
        assert H.TriangleCounting2(h).run() == O.tc(g)
    finally:
        H.tune_reset()


@pytest.mark.parametrize("case", ["union", "small", "one_tile", "hub"])
def test_close_ids_use_bitmaps_of_ids(case):
    """Lists under ids that span less than a warp's bitmap (65,536 ids), than
    a CTA's (131,072), and more; one vertex's list across many tiles."""
    rng = np.random.default_rng(8)
    if case == "union":
        parts = [T.rmat_graph(13, 16, seed=1), T.er_graph(90_000, 40, seed=2),
                 T.rmat_graph(17, 8, seed=3, n_vertices=70_001), T.er_graph(300, 150, seed=4),
                 T.er_graph(140_000, 12, seed=9)]
        g, _ = T.disjoint_union(parts)
    elif case == "small":
        g = T.rmat_graph(10, 40, seed=5)
    elif case == "one_tile":
        g = T.er_graph(40, 9, seed=6)
    else:
        n = 40_000       # two vertices joined to nearly all, which form short lists
        a = rng.permutation(n)[:39_000].astype(np.int32)
        s = [np.full(39_000, 7, np.int32), np.full(39_000, 39_991, np.int32), a[:-1]]
        d = [a, a[::-1].copy(), a[1:]]
        s, d = np.concatenate(s), np.concatenate(d)
        keep = s != d
        g = O.build_csr_undirected(n, s[keep], d[keep])
    h = build(g)
    ref = O.tc(g)
    tc = H.TriangleCounting2(h)
    for knobs in ({}, {"tc.warp_cap": 32, "tc.warp_work": 1024, "tc.mid_cap": 32,
                       "tc.item_work": 1024}, {"tc.thread_du": 0}):
        try:
            for k, v in knobs.items():
                H.tune_set(k, v)
            assert tc.run() == ref
            assert tc.run(per_vertex=True) == ref
            pv = tc.copyTCToHost().copy()
            ow, total = owner(h)
            assert total == ref == int(ow.sum())
            H.tune_set("tc.flip", 0)
            assert tc.run(per_vertex=True) == ref
            np.testing.assert_array_equal(pv, tc.copyTCToHost())
            ow0, _ = owner(h)
            np.testing.assert_array_equal(ow, ow0)
        finally:
            H.tune_reset()


def test_a_busy_handle_is_refused():
    """Owner counts called on a handle that another thread is counting on:
    each call returns the counts or HN_ERR_STATE."""
    import threading
    g = T.rmat_graph(18, 16, seed=7)
    h = build(g)
    ref = O.tc(g)
    assert owner(h)[1] == ref
    codes, wrong, start = [], [], threading.Barrier(2)

    def count():
        start.wait()
        for _ in range(50):
            try:
                if owner(h)[1] != ref:
                    wrong.append(1)
                codes.append(0)
            except H.HornetError as e:
                codes.append(e.code)

    threads = [threading.Thread(target=count) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong and set(codes) == {0, H.HN_ERR_STATE}
    assert owner(h)[1] == ref
