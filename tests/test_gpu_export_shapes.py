"""Exports (COO, CSR, weights) at the sizes where a warp tile or a prefix-sum
chunk ends: runs of empty vertices, one vertex spanning many tiles, tiles of
256 and 1024 elements with remainders, vertex counts around the one-kernel
prefix sum's chunk and limit."""
import numpy as np
import pytest

import hornet_b200 as H

pytestmark = pytest.mark.gpu


def csr_of(deg):
    """A sorted directed CSR with these out-degrees (each at most nV)."""
    deg = np.asarray(deg, np.int64)
    off = np.concatenate([[0], np.cumsum(deg)])
    seg = np.repeat(np.arange(len(deg)), deg)
    adj = (np.arange(off[-1]) - off[seg]).astype(np.int32)   # 0..deg-1 of each vertex
    return off.astype(np.int32), adj, seg.astype(np.int32)


def degrees(kind):
    rng = np.random.default_rng(7)
    if kind == "empty_runs":        # edges only at both ends and in the middle
        d = np.zeros(50_000, np.int64)
        d[[0, 25_000, 49_999]] = [3, 1, 700]
        return d
    if kind == "one_hub":           # a vertex spanning many tiles between small ones
        d = rng.integers(0, 3, 9000)
        d[4321] = 8999
        return d
    if kind == "all_ones":
        return np.ones(4099, np.int64)
    if kind == "remainders":        # segments around the row and window lengths
        return np.tile([0, 1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 0, 0], 40)
    if kind == "isolated":
        return np.zeros(1000, np.int64)
    return rng.integers(0, 40, 60_000)


@pytest.mark.parametrize("kind", ["empty_runs", "one_hub", "all_ones", "remainders", "isolated",
                                  "random"])
@pytest.mark.parametrize("weighted", [False, True])
def test_export_matches_csr(kind, weighted):
    off, adj, seg = csr_of(degrees(kind))
    init = H.HornetInit(len(off) - 1, len(adj), off, adj, sorted_adjacency=True)
    w = (np.arange(len(adj)) * 7 + 3).astype(np.uint32)
    if weighted:
        init.insertEdgeData(w)
    h = H.Hornet(init)
    s, d = h.getCOO(True)
    np.testing.assert_array_equal(s, seg)
    np.testing.assert_array_equal(d, adj)
    o2, a2 = h.getCSR()
    np.testing.assert_array_equal(o2, off)
    np.testing.assert_array_equal(a2, adj)
    if weighted:
        s, d, w2 = h.getCOOWeighted()
        np.testing.assert_array_equal(s, seg)
        np.testing.assert_array_equal(d, adj)
        np.testing.assert_array_equal(w2, w)


@pytest.mark.parametrize("nV", [1, 2, 8191, 8192, 8193, 16383, 16384, 65537])
def test_export_at_prefix_sum_sizes(nV):
    rng = np.random.default_rng(nV)
    off, adj, seg = csr_of(np.minimum(rng.integers(0, 5, nV), nV))
    h = H.Hornet(H.HornetInit(nV, len(adj), off, adj, sorted_adjacency=True))
    s, d = h.getCOO(True)
    np.testing.assert_array_equal(s, seg)
    np.testing.assert_array_equal(d, adj)


def test_export_with_large_tiles():
    """More edges than the 256-element tiles are used for."""
    rng = np.random.default_rng(5)
    n = 600_000
    d = np.minimum((rng.pareto(1.1, n) * 30).astype(np.int64), 20_000)
    d[rng.random(n) < 0.4] = 0
    d[n // 2] = 400_000
    while d.sum() < 42_000_000:
        d[rng.integers(0, n, 1000)] += 500
    off, adj, seg = csr_of(d)
    h = H.Hornet(H.HornetInit(n, len(adj), off, adj, sorted_adjacency=True))
    s, dd = h.getCOO(True)
    assert (s == seg).all() and (dd == adj).all()
