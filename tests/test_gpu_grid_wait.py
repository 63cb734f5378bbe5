"""Waits of the cooperative launches (one-launch BFS, k-truss rounds) that run
out: the limit is set to a quarter of a millisecond and one warp or CTA has
a long list to read while the others wait.  The call
reports HN_ERR_TIMEOUT, and the next call on the handle is right."""
import numpy as np
import pytest

import hornet_b200 as H
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIRST = 3000   # neighbours of the source, each with two more


def device_graph(n, s, d):
    import torch
    s, d = (torch.from_numpy(np.ascontiguousarray(x, np.int32)).cuda() for x in (s, d))
    torch.cuda.synchronize()
    return H.hornet_from_device_csr(H.coo_to_csr_device(n, s, d))


def hub_off_the_frontier(leaves):
    """Vertex 0 with FIRST neighbours, each with two more; apart from them a
    hub, which a bottom-up level reads to its end.  Distances from 0."""
    kids = 1 + np.arange(FIRST)
    grand = 1 + FIRST + np.arange(2 * FIRST)
    hub = 1 + 3 * FIRST
    s = np.concatenate([np.zeros(FIRST), np.repeat(kids, 2), np.full(leaves, hub)])
    d = np.concatenate([kids, grand, hub + 1 + np.arange(leaves)])
    dist = np.full(hub + 1 + leaves, O.INF, np.int32)
    dist[0], dist[kids], dist[grand] = 0, 1, 2
    return device_graph(len(dist), s, d), dist


def double_star(leaves):
    """Two joined hubs without a common neighbour: no triangle, one edge with
    a long intersection."""
    s = np.concatenate([[0], np.zeros(leaves), np.ones(leaves)])
    d = np.concatenate([[1], 2 + np.arange(2 * leaves)])
    return device_graph(2 + 2 * leaves, s, d)


BOTTOM_UP = {"bfs.do_alpha": 1 << 20, "bfs.do_beta": 1 << 20}


def test_bfs_wait_gives_up():
    import torch
    h, dist = hub_off_the_frontier(1_000_000)
    out = torch.empty((8, len(dist)), dtype=torch.int32, device="cuda:0")
    bfs = H.BfsTopDown(h)
    try:
        for k, v in BOTTOM_UP.items():
            H.tune_set(k, v)
        for _ in range(2):
            H.tune_set("grid.wait_polls", 1024)
            # the sources behind the first are queued when its wait gives up
            with pytest.raises(H.HornetError) as e:
                bfs.run_multi([0] * 8, out=out, direction_optimizing=True)
            assert e.value.code == H.HN_ERR_TIMEOUT
            H.tune_set("grid.wait_polls", 1 << 24)
            out.fill_(-1)
            torch.cuda.synchronize()
            _, st = bfs.run_multi([0] * 8, out=out, direction_optimizing=True)
            for i in range(8):
                np.testing.assert_array_equal(out[i].cpu().numpy(), dist)
                assert st[i].visited == 1 + 3 * FIRST and st[i].levels == 3
    finally:
        H.tune_reset()


def test_bfs_wait_gives_up_with_copies_queued():
    """Distances to pinned host memory: when the call has reported the error,
    no copy into the caller's array is still to come."""
    import torch
    h, dist = hub_off_the_frontier(1_000_000)
    out = torch.empty((70, len(dist)), dtype=torch.int32, pin_memory=True).numpy()
    bfs = H.BfsTopDown(h)
    try:
        for k, v in BOTTOM_UP.items():
            H.tune_set(k, v)
        H.tune_set("grid.wait_polls", 1024)
        with pytest.raises(H.HornetError) as e:
            bfs.run_multi([0] * 70, out=out, direction_optimizing=True)
        out[:, -1] = -7
        assert e.value.code == H.HN_ERR_TIMEOUT
        torch.cuda.synchronize()
        assert (out[:, -1] == -7).all()
        H.tune_set("grid.wait_polls", 1 << 24)
        bfs.run_multi([0] * 70, out=out, direction_optimizing=True)
        for i in (0, 1, 63, 64, 69):
            np.testing.assert_array_equal(out[i], dist)
    finally:
        H.tune_reset()


def test_slow_work_is_progress():
    """A warp that reads 4 M neighbours (37 ms), and a CTA that intersects lists
    of 8 M (28 ms), take longer than the limit (about 9 ms) but tell the others
    every 1.2 and 2 ms that they go on."""
    h, dist = hub_off_the_frontier(4_000_000)
    try:
        for k, v in BOTTOM_UP.items():
            H.tune_set(k, v)
        H.tune_set("grid.wait_polls", 1 << 15)
        out, _ = H.BfsTopDown(h).run_multi([0], direction_optimizing=True)
        np.testing.assert_array_equal(out[0], dist)
        kt = H.KTruss(double_star(8_000_000))
        assert kt.run() == 2
        assert (kt.edge_truss == 2).all()
    finally:
        H.tune_reset()


def test_ktruss_wait_gives_up():
    h = double_star(4_000_000)
    kt = H.KTruss(h)
    try:
        H.tune_set("grid.wait_polls", 1024)
        with pytest.raises(H.HornetError) as e:
            kt.run()
        assert e.value.code == H.HN_ERR_TIMEOUT
    finally:
        H.tune_reset()
    assert kt.run() == 2
    assert (kt.edge_truss == 2).all()
