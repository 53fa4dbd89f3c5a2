"""The flat pull (edge streams cut into steps and pieces) at the sizes where
its cuts fall: a step of 256 cold or 512 hot edges and one more or less, the
one-CTA limit of the one-launch epochs, rows longer than a piece, rows without
edges, graphs on both sides of the one-launch limit and with hot streams.
Ranks against the double-precision oracle: L1 <= 1e-6 (normalised), the
library's bar for 32-bit ranks; epochs equal."""
import numpy as np
import pytest

import plato_b200 as pb
from oracle import RefGraph, fp64

pytestmark = pytest.mark.gpu


def _random(V, E, seed, hub=0.0):
    """E directed edges over V vertices, a share `hub` of them into vertex 1."""
    rng = np.random.default_rng(seed)
    s = rng.integers(0, V, E, dtype=np.uint32)
    d = rng.integers(0, V, E, dtype=np.uint32)
    d[rng.random(E) < hub] = 1
    return V, s, d


GRAPHS = [(2, 1, 0.0), (33, 255, 0.0), (33, 256, 0.5), (64, 257, 0.0), (2, 300, 1.0), (100, 16384, 0.0),
          (1000, 16640, 0.9), (3001, 40000, 0.3), (70001, 100000, 0.0), (5, 70000, 1.0), (200003, 3499999, 0.05),
          (200003, 3500001, 0.05)]


@pytest.mark.parametrize("V,E,hub", GRAPHS)
@pytest.mark.parametrize("early", [False, True])
def test_pagerank_at_the_cuts(V, E, hub, early):
    """The early exit at a delta of 1e-6 (normalised): 32-bit ranks round their
    deltas by up to 2^-24 in sum, so the epochs agree within one."""
    V, s, d = _random(V, E, 7 * V + E, hub)
    eps = 1e-6 * V if early else 0.0
    want, epochs, _ = RefGraph(V, s, d, True).pagerank(15 if eps == 0 else 100, 0.85, eps)
    with pb.Graph(V, s, d, True) as g:
        got, st = g.pagerank(15 if eps == 0 else 100, 0.85, eps)
        again, _ = g.pagerank(15 if eps == 0 else 100, 0.85, eps)
    assert abs(st.iterations - epochs) <= (0 if eps == 0 else 1)
    assert np.abs(got.astype(np.float64) - want / V).sum() <= 1e-6
    np.testing.assert_array_equal(got, again)  # the same from run to run


@pytest.mark.parametrize("iteration", [1, 2, 3, 20])
@pytest.mark.parametrize("graph", ["rmat19", "uniform"])
def test_hot_streams(graph, iteration):
    """Above 8M edges out of the first 57344 sources the pull has hot streams;
    the uniform graph's rows are long enough to take part in all of them."""
    if graph == "rmat19":
        V, s, d = pb.rmat(19, 24, 3)
    else:
        V, s, d = _random(120001, 20000000, 5, 0.01)
    want, epochs, _ = RefGraph(V, s, d, True).pagerank(iteration, 0.85, 0.0)
    with pb.Graph(V, s, d, True) as g:
        got, st = g.pagerank(iteration, 0.85, 0.0)
        again, _ = g.pagerank(iteration, 0.85, 0.0)
    assert st.iterations == epochs
    assert np.abs(got.astype(np.float64) - want / V).sum() <= 1e-6
    np.testing.assert_array_equal(got, again)


@pytest.mark.parametrize("edges", [3000, 12000000])
@pytest.mark.parametrize("early", [False, True])
def test_weighted(edges, early):
    V = 400 if edges < 10000 else 100003
    V, s, d = _random(V, edges, 11, 0.02)
    eps = 1e-6 * V if early else 0.0
    w = np.random.default_rng(1).uniform(0.1, 10, edges)
    want, epochs, _ = fp64.weighted_pagerank(V, s, d, w, True, 60, 0.85, eps)
    with pb.Graph(V, s, d, True, weights=w) as g:
        got, st = g.weighted_pagerank(60, 0.85, eps)
    assert abs(st.iterations - epochs) <= (0 if eps == 0 else 1)
    assert np.abs(got - want).sum() / V <= 1e-6


@pytest.mark.parametrize("edges", [5000, 12000000])
def test_not_a_number_stays_in_its_rows(edges):
    """A vertex whose out-weights are all 0 gathers as inf: its targets become
    NaN in the first epoch, no other row does."""
    V = 900 if edges < 10000 else 100003
    V, s, d = _random(V, edges, 13)
    w = np.ones(edges)
    w[s == 3] = 0.0
    hit = np.zeros(V, bool)
    hit[d[s == 3]] = True
    with pb.Graph(V, s, d, True, weights=w) as g:
        got, _ = g.weighted_pagerank(1, 0.85, 0.0)
    np.testing.assert_array_equal(np.isnan(got), hit)


@pytest.mark.parametrize("scale", [10, 19])
def test_seed_sets_and_single_queries(scale):
    V, s, d = pb.rmat(scale, 24, 8)
    ref = RefGraph(V, s, d, True)
    deg = np.bincount(s, minlength=V)
    src = int(np.argmax(deg))
    with pb.Graph(V, s, d, True) as g:
        for mode, dual in ((pb.PLATO_PPR_PULL, False), (pb.PLATO_PPR_PUSHPULL, True)):
            got, st = g.personalized_pagerank(src, 100, 0.85, 1e-6, mode)
            want, epochs = ref.ppr(src, 100, 0.85, 1e-6, dual)[:2]
            assert abs(st.iterations - epochs) <= 1
            # the bar, and one epoch that moves less than eps where one side ends earlier
            assert np.abs(got.astype(np.float64) - want).sum() <= 1e-6 + 1e-6


@pytest.mark.parametrize("E", [11 << 20, 16 << 20])
def test_cold_stream_waves(E):
    """One wave of cold pieces, taken in order, and more, taken from the end."""
    V, s, d = _random(1000003, E, 11, 0.01)
    want, _, _ = RefGraph(V, s, d, True).pagerank(5, 0.85, 0.0)
    with pb.Graph(V, s, d, True) as g:
        got, _ = g.pagerank(5, 0.85, 0.0)
        again, _ = g.pagerank(5, 0.85, 0.0)
    assert np.abs(got.astype(np.float64) - want / V).sum() <= 1e-6
    np.testing.assert_array_equal(got, again)


def test_no_room_for_the_plan():
    """With less memory left than the plan takes (RMAT s20: 50 MB and its
    scratch) the merge path answers; a later graph gets its plan again."""
    import torch

    V, s, d = pb.rmat(20, 16, 9)
    want, epochs, _ = RefGraph(V, s, d, True).pagerank(10, 0.85, 0.0)
    with pb.Graph(1000, s[:100] % 1000, d[:100] % 1000, True, relabel=False) as small:
        small.pagerank(2, 0.85, 0.0)  # the merge path's kernels are loaded
    with pb.Graph(V, s, d, True) as g:
        free, _ = torch.cuda.mem_get_info()
        hog = torch.empty(max(free - (32 << 20), 0), dtype=torch.uint8, device="cuda")
        try:
            got, st = g.pagerank(10, 0.85, 0.0)
        finally:
            del hog
            torch.cuda.empty_cache()
        again, _ = g.pagerank(10, 0.85, 0.0)
    assert st.iterations == epochs
    assert np.abs(got.astype(np.float64) - want / V).sum() <= 1e-6
    np.testing.assert_array_equal(got, again)  # the graph stays on its path
