"""k-truss peel rounds at the edges of their three forms: frontiers of one
CTA (16 edges), staged by every CTA (512) and split over the CTAs, the
largest with several stagings a CTA; next to a graph with long rounds."""
import numpy as np
import pytest

import hornet_b200 as H
from oracle import oracle as O
from tests import helpers as T

pytestmark = pytest.mark.gpu


def graph(n):
    """n edges without a triangle (the frontier of K = 3), a strip of n
    triangles (peeled from its two ends at K = 4, two rounds' frontiers of a
    few edges at a time when n is small; all n when cut into single
    triangles) and a K6 on scattered ids, beside an R-MAT graph."""
    core = T.rmat_graph(9, 8, seed=5)
    s = [np.repeat(np.arange(core.nV), np.diff(core.off)), ]
    d = [core.adj]
    at = core.nV
    e = np.arange(n)
    s.append(at + 2 * e)             # single edges
    d.append(at + 2 * e + 1)
    at += 2 * n
    for x, y in ((0, 1), (1, 2), (0, 2)):   # single triangles
        s.append(at + 3 * e + x)
        d.append(at + 3 * e + y)
    at += 3 * n
    m = min(n, 600)
    for step in (1, 2):              # a strip of triangles
        i = np.arange(m)
        s.append(at + i)
        d.append(at + i + step)
    at += m + 2
    k = at + 7 * np.arange(6)
    s.append(np.repeat(k, 6))
    d.append(np.tile(k, 6))
    at = int(k[-1]) + 1
    s, d = np.concatenate(s).astype(np.int32), np.concatenate(d).astype(np.int32)
    keep = s != d
    return O.build_csr_undirected(at, s[keep], d[keep])


@pytest.mark.parametrize("n", [1, 5, 6, 16, 17, 64, 65, 171, 512, 513, 3000, 90_000])
def test_frontiers(n):
    g = graph(n)
    h = H.Hornet(H.HornetInit(g.nV, g.nE, g.off32(), g.adj, sorted_adjacency=True))
    kt = H.KTruss(h)
    kmax, et = O.ktruss_peel(g)
    assert kt.run() == kmax
    np.testing.assert_array_equal(kt.edge_truss, et)
