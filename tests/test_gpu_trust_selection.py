"""Seed selection on the flat pull in 64 bits: one launch (small graphs), three
kernels an epoch, and hot streams; over the in-edges and the out-edges, whose
rows are in no order of their degree; both vertex orders.  The seeds equal the
ones a 64-bit PageRank picks wherever its ranks at the cut differ by more than
1e-9 relative; a graph without edges keeps its first vertices."""
import numpy as np
import pytest

import plato_b200 as pb
from oracle import fp64

pytestmark = pytest.mark.gpu


def _select(V, s, d, inverse, n):
    r, _ = fp64.pagerank(V, d if inverse else s, s if inverse else d, True, 100, 0.85, 0.001)
    order = np.lexsort((np.arange(V), -r))
    return order, r


@pytest.mark.parametrize("method", [0, 1])
@pytest.mark.parametrize("relabel", [True, False])
@pytest.mark.parametrize("scale,ef", [(7, 8), (11, 16), (17, 40), (19, 30)])
def test_seeds(scale, ef, relabel, method):
    V, s, d = pb.rmat(scale, ef, 5)
    order, r = _select(V, s, d, method == 0, 50)
    with pb.Graph(V, s, d, True, relabel=relabel) as g:
        for n in (1, 40):
            cut = (r[order[n - 1]] - r[order[n]]) / r[order[n]]
            ranks, seeds, _ = g.trustrank(None, 30, 0.85, n, method, 0.0)
            again = g.trustrank(None, 30, 0.85, n, method, 0.0)
            if cut > 1e-9:
                np.testing.assert_array_equal(seeds, np.sort(order[:n]).astype(np.uint32))
            np.testing.assert_array_equal(seeds, again[1])
            np.testing.assert_array_equal(ranks, again[0])
            want, _ = fp64.seedset_ppr(V, s, d, seeds, True, 30, 0.85, 0.0)
            assert np.abs(ranks - want).sum() <= 1e-6


def test_no_edges():
    s = np.array([], np.uint32)
    with pb.Graph(9, s, s, True) as g:
        _, seeds, _ = g.trustrank(None, 5, 0.85, 3, 0, 0.0)
    np.testing.assert_array_equal(seeds, [0, 1, 2])
