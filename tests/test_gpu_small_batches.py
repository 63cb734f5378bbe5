"""Updates at the sizes where the batch pipeline changes: the one-CTA front
for up to 2,048 entries (and the sort network's powers of two), with and
without touched hubs, every combination of de-duplication flags, block-class
changes, emptied vertices; coalesced runs on both sides of the limit."""
import numpy as np
import pytest

import hornet_b200 as H
from oracle import oracle as O
from tests import helpers as T

pytestmark = pytest.mark.gpu


def build(g):
    return H.Hornet(H.HornetInit(g.nV, g.nE, g.off32(), g.adj, sorted_adjacency=True))


def assert_equal(h, g):
    s, d = h.getCOO(True)
    es, ed = g.coo()
    np.testing.assert_array_equal(s, es)
    np.testing.assert_array_equal(d, ed)


@pytest.mark.parametrize("hubs", [False, True])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1000, 1023, 1024, 1025, 2047, 2048, 2049, 4096])
def test_small_batches(n, hubs):
    """hubs: half of the entries hit the vertices of highest degree (over the
    hub threshold, lowered to 64)."""
    g = T.rmat_graph(11, 16, seed=4)
    h = build(g)
    rng = np.random.default_rng(n + hubs)
    deg = np.diff(g.off)
    top = np.argsort(-deg)[:3].astype(np.int32)
    try:
        if hubs:
            H.tune_set("update.big_min", 64)
        for flags in range(4):
            bs = rng.integers(0, g.nV, n).astype(np.int32)
            bd = rng.integers(0, g.nV, n).astype(np.int32)
            if hubs:
                bs[::2] = top[rng.integers(0, 3, len(bs[::2]))]
            bs[n // 2:n // 2 + n // 8], bd[n // 2:n // 2 + n // 8] = bs[:n // 8], bd[:n // 8]
            added = h.insert(H.BatchUpdate(h, bs, bd), bool(flags & 1), bool(flags & 2))
            g, ref = O.insert(g, bs, bd, flags)
            assert added == ref
            assert_equal(h, g)
            es, ed = g.coo()
            sel = rng.integers(0, len(es), n)
            xs, xd = es[sel].copy(), ed[sel].copy()
            xs[::5] = bs[::5]
            xd[::5] = bd[::5]
            removed = h.erase(H.BatchUpdate(h, xs, xd), bool(flags & 1))
            g, ref = O.erase(g, xs, xd, flags & 1)
            assert removed == ref
            assert_equal(h, g)
    finally:
        H.tune_reset()


def test_small_batch_empties_and_refills_a_vertex():
    g = T.rmat_graph(9, 8, seed=6)
    h = build(g)
    deg = np.diff(g.off)
    u = int(np.argsort(-deg)[5])
    nb = g.adj[g.off[u]:g.off[u + 1]].copy()
    src = np.full(len(nb), u, np.int32)
    assert h.erase(H.BatchUpdate(h, src, nb), True) == len(nb)
    g2, _ = O.erase(g, src, nb, 1)
    assert_equal(h, g2)
    assert h.insert(H.BatchUpdate(h, src[::-1].copy(), nb[::-1].copy()), True, True) == len(nb)
    assert_equal(h, g)


def test_small_batch_with_a_bad_id_is_refused():
    g = T.rmat_graph(9, 8, seed=6)
    h = build(g)
    for bad in (-1, g.nV):
        with pytest.raises(H.HornetError) as e:
            h.insert(H.BatchUpdate(h, np.array([1, bad], np.int32), np.array([2, 3], np.int32)))
        assert e.value.code == H.HN_ERR_INVALID
    assert_equal(h, g)


@pytest.mark.parametrize("n", [1, 500, 3000, 20_000])
def test_coalesced_runs(n):
    g = T.rmat_graph(12, 8, seed=8)
    h = build(g)
    rng = np.random.default_rng(n)
    es, ed = g.coo()
    sel = rng.integers(0, len(es), n)
    src = np.concatenate([es[sel], rng.integers(0, g.nV, n).astype(np.int32), es[sel[:n // 3]]])
    dst = np.concatenate([ed[sel], rng.integers(0, g.nV, n).astype(np.int32), ed[sel[:n // 3]]])
    ops = np.concatenate([np.zeros(n), np.ones(n), np.ones(n // 3)]).astype(np.uint8)
    ins, era = h.update_coalesced(src, dst, ops)
    last = {}
    for a, b, o in zip(src.tolist(), dst.tolist(), ops.tolist()):
        last[(a, b)] = o
    have = set(zip(es.tolist(), ed.tolist()))
    add = {e for e, o in last.items() if o and e not in have}
    rem = {e for e, o in last.items() if not o and e in have}
    assert (ins, era) == (len(add), len(rem))
    want = np.array(sorted((have - rem) | add), np.int64)
    s, d = h.getCOO(True)
    np.testing.assert_array_equal(s, want[:, 0])
    np.testing.assert_array_equal(d, want[:, 1])
