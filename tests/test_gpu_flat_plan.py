"""The flat pull's reports and plans at the edges of what takes it: the delta
of a call whose only pull epoch is the final one, and graphs whose rows,
sources or memory do not suit a flat plan."""
import ctypes as C

import numpy as np
import pytest

import plato_b200 as pb
from oracle import RefGraph, fp64
from plato_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,ef", [(10, 16), (14, 16), (18, 20)])
def test_delta_of_the_push_epochs_outlives_a_final_pull(scale, ef):
    """A hub's neighbours switch the query to pull in its second and last
    epoch, which has no delta: the push epoch's is reported, on both sides of
    the one-launch limit (3.5M edges), whatever an earlier call left."""
    V, s, d = pb.rmat(scale, ef, 3)
    ref = RefGraph(V, s, d, True)
    src = int(np.argmax(np.bincount(s, minlength=V)))
    with pb.Graph(V, s, d, True) as g:
        g.pagerank(4, 0.85, 1e-9)  # another call's delta on the same graph
        _, st = g.personalized_pagerank(src, 2, 0.85, 1e-9, pb.PLATO_PPR_PUSHPULL)
        one = g.pagerank(1, 0.85, 1e-9)[1]
    _, epochs, pushes, _, delta = ref.ppr(src, 2, 0.85, 1e-9, True)
    assert (st.iterations, st.push_iterations) == (epochs, pushes) == (2, 1)
    assert delta > 1.0 and st.delta == pytest.approx(delta, rel=1e-5)  # 32-bit terms, 2^-24 each
    assert one.delta == 0.0  # no epoch with a delta ran


@pytest.mark.parametrize("scale", [10, 18])
def test_delta_with_an_eps_that_is_no_number(scale):
    """NaN ends no epoch early and asks for the deltas, as an eps that no delta
    reaches does: the same ranks and the same delta, also after other calls."""
    V, s, d = pb.rmat(scale, 20, 5)
    with pb.Graph(V, s, d, True) as g:
        want, ws = g.pagerank(6, 0.85, 1e-300)
        g.pagerank(20, 0.85, 1e-300)  # leaves a smaller delta
        got, st = g.pagerank(6, 0.85, float("nan"))
    np.testing.assert_array_equal(got, want)
    assert (st.iterations, st.delta) == (ws.iterations, ws.delta)


def test_a_barrier_that_runs_out_is_an_error():
    """With no polls allowed the blocks of the one-launch epochs give up at
    their first barrier: every rank call that hands out host ranks says so,
    with and without an early exit, and the graph answers again afterwards."""
    V, s, d = pb.rmat(15, 16, 6)
    w = np.random.default_rng(2).uniform(0.1, 10, s.size)
    lib = _lib.load()
    src = int(s[0])

    def calls(g, eps):
        return [lambda: g.pagerank(10, 0.85, eps)[0],
                lambda: g.weighted_pagerank(10, 0.85, eps)[0],
                lambda: g.personalized_pagerank(src, 10, 0.85, eps, pb.PLATO_PPR_PULL)[0],
                lambda: g.personalized_pagerank(src, 10, 0.85, eps, pb.PLATO_PPR_PUSHPULL)[0],
                lambda: g.seedset_ppr([src, 1], 10, 0.85, eps)[0]]

    with pb.Graph(V, s, d, True, weights=w) as g:
        for eps in (0.0, 1e-9):
            want = [call() for call in calls(g, eps)]
            _lib.check(lib.plato_diag_barrier_polls(g.handle, 0), "polls")
            for call in calls(g, eps):
                with pytest.raises(_lib.PlatoError) as e:
                    call()
                assert e.value.code == _lib.PLATO_ETIMEDOUT
            _lib.check(lib.plato_diag_barrier_polls(g.handle, 1 << 24), "polls")
            for call, ranks in zip(calls(g, eps), want):
                # the push epochs add in any order
                np.testing.assert_allclose(call(), ranks, rtol=0, atol=1e-6 * ranks.max())
    assert lib.plato_diag_barrier_polls(None, 0) == _lib.PLATO_EINVAL


def _launched(call, names):
    """The kernels among `names` that `call` launches, and its result."""
    lib = _lib.load()
    _lib.check(lib.plato_profile_enable(1), "profile")
    _lib.check(lib.plato_profile_reset(), "profile")
    try:
        out = call()
    finally:
        lib.plato_profile_enable(0)
    hit = set()
    for n in names:
        ms, k = C.c_double(), C.c_uint64()
        _lib.check(lib.plato_profile_read(n.encode(), C.byref(ms), C.byref(k)), n)
        if k.value:
            hit.add(n)
    return hit, out


KERNELS = ["k_flat_hot", "k_flat_cold", "k_flat_update", "k_flat_run", "k_pull_long", "k_pull_rows16", "k_pull_rows8",
           "k_pull_rows4", "k_pull_short", "k_pull_hubs", "k_pull_warp"]


@pytest.mark.parametrize("weighted", [False, True])
def test_bins_answer_without_room_for_the_plan(weighted):
    """With 32 MB left the flat plan of RMAT s20 does not fit and the degree
    bins answer, weights and early exit too; the graph stays with them when the
    memory comes free, and the next graph gets its plan."""
    import torch

    V, s, d = pb.rmat(20, 16, 9)
    w = np.random.default_rng(3).uniform(0.1, 10, s.size) if weighted else None

    def call(g, eps=0.0):
        return g.weighted_pagerank(12, 0.85, eps) if weighted else g.pagerank(12, 0.85, eps)

    eps = 2e-2 * V
    with pb.Graph(V, s, d, True, weights=w) as g:
        plan, (want, _) = _launched(lambda: call(g), KERNELS)
        want_early, early = call(g, eps)
        assert "k_flat_cold" in plan and not any(n.startswith("k_pull") for n in plan)
        assert early.iterations < 12
    with pb.Graph(V, s, d, True, weights=w) as g:
        free, _ = torch.cuda.mem_get_info()
        hog = torch.empty(max(free - (32 << 20), 0), dtype=torch.uint8, device="cuda")
        try:
            bins, (got, _) = _launched(lambda: call(g), KERNELS)
            got_early, st = call(g, eps)
        finally:
            del hog
            torch.cuda.empty_cache()
        later, (again, _) = _launched(lambda: call(g), KERNELS)
        with pb.Graph(V, s, d, True, weights=w) as g2:
            fresh, (new, _) = _launched(lambda: call(g2), KERNELS)
    assert {"k_pull_long", "k_pull_short"} <= bins and bins == later
    assert not any(n.startswith("k_flat") or n == "k_pull_warp" for n in bins)
    assert fresh == plan
    unit = V if weighted else 1  # sums of 32-bit ranks in two orders, each within 1e-6 of the oracle's
    assert np.abs(got.astype(np.float64) - want).sum() / unit <= 2e-6
    assert np.abs(got_early.astype(np.float64) - want_early).sum() / unit <= 2e-6
    assert st.iterations == early.iterations and st.delta == pytest.approx(early.delta, rel=1e-3)
    np.testing.assert_array_equal(again, got)
    np.testing.assert_array_equal(new, want)


def test_a_graph_without_edges_takes_the_bins():
    V = 70001
    with pb.Graph(V, np.zeros(0, np.uint32), np.zeros(0, np.uint32), True) as g:
        hit, (got, st) = _launched(lambda: g.pagerank(4, 0.85, 0.0), KERNELS)
    assert hit == {"k_pull_short"} and st.iterations == 4
    np.testing.assert_allclose(got, 0.15 / V, rtol=1e-6)


def test_device_bytes_count_the_plan_and_the_index():
    """The flat plan holds every edge once more, 2 bytes (hot) or 4 (cold), and
    the components' index the non-empty columns' starts."""
    V, s, d = pb.rmat(18, 16, 4)
    with pb.Graph(V, s, d, True) as g:
        E = g.device_view().stored_edges
        plain = g.device_bytes()
        g.pagerank(2, 0.85, 0.0)
        ranked = g.device_bytes()
        assert 2 * E <= ranked - plain <= 6 * E
        g.pagerank(2, 0.85, 0.0)
        assert g.device_bytes() == ranked  # kept, not built again
        g.connected_components()
        columns = np.unique(d).size
        assert g.device_bytes() - ranked >= 12 * columns


@pytest.mark.parametrize("V,E,share", [(40, 20000, 1.0), (1000, 300000, 0.5), (100003, 3000000, 1.0),
                                       (100003, 4000000, 1.0), (1000003, 5000000, 0.9), (200003, 12000000, 0.7),
                                       (1500007, 20000000, 0.5)])
def test_rows_across_many_pieces(V, E, share):
    """A vertex with most of the in-edges crosses every piece of its streams:
    on the one-launch path, in the cold stream, where all sources are hot, and
    in both kinds of stream.  L1 <= 1e-6, and the same from run to run."""
    rng = np.random.default_rng(E)
    s = rng.integers(0, V, E, dtype=np.uint32)
    d = rng.integers(0, V, E, dtype=np.uint32)
    d[rng.random(E) < share] = 1
    want, _, _ = RefGraph(V, s, d, True).pagerank(6, 0.85, 0.0)
    with pb.Graph(V, s, d, True) as g:
        got, _ = g.pagerank(6, 0.85, 0.0)
        again, _ = g.pagerank(6, 0.85, 0.0)
    assert np.abs(got.astype(np.float64) - want / V).sum() <= 1e-6
    np.testing.assert_array_equal(got, again)


def _uniform(V, E):
    rng = np.random.default_rng(V + E)
    return V, rng.integers(0, V, E, dtype=np.uint32), rng.integers(0, V, E, dtype=np.uint32)


@pytest.mark.parametrize("V,E", [(8192, 8), (8193, 8), (300007, 8), (1000003, 500000), (6000000, 900000),
                                 (6000001, 900000)])
def test_few_edges_over_many_rows(V, E):
    """The warps of the one-launch epochs follow the rows too, up to 6M of
    them; with a first row that is long, so that no shorter way answers."""
    _, s, d = _uniform(V, E)
    s, d = np.append(s, np.arange(600, dtype=np.uint32)), np.append(d, np.full(600, 5, np.uint32))
    want, _, _ = RefGraph(V, s, d, True).pagerank(5, 0.85, 0.0)
    with pb.Graph(V, s, d, True) as g:
        hit, (got, _) = _launched(lambda: g.pagerank(5, 0.85, 0.0), KERNELS)
        ms, n = C.c_double(), C.c_uint64()
        if V <= 1000003:  # by the edges alone 300007 rows took 0.9 ms an epoch
            lib = _lib.load()
            assert hit == {"k_flat_run"}
            _lib.check(lib.plato_profile_read(b"k_flat_run", C.byref(ms), C.byref(n)), "read")
            assert n.value == 1 and ms.value < 1.0
    assert np.abs(got.astype(np.float64) - want / V).sum() <= 1e-6


def _ring(V):
    i = np.arange(V, dtype=np.uint32)
    return V, i, (i + 1) % np.uint32(V)


def _capped(V, k):
    """k in-edges for every vertex but one, which has none."""
    rng = np.random.default_rng(V + k)
    d = np.repeat(np.arange(V, dtype=np.uint32), k)
    s = rng.integers(0, V, d.size, dtype=np.uint32)
    return V, s[d != 0], d[d != 0]


ONE, TWO = {"k_pull_short"}, {"k_pull_short", "k_pull_rows4"}
RUN, COLD = {"k_flat_run"}, {"k_flat_cold", "k_flat_update"}


@pytest.mark.parametrize("graph,kernels", [
    (_ring(8192), RUN), (_ring(8193), ONE), (_ring(100003), ONE), (_capped(8193, 4), ONE), (_capped(8193, 5), RUN), (_capped(900001, 4), ONE),
    (_uniform(1000003, 1000), ONE), (_uniform(1000003, 500000), RUN), (_uniform(1000003, 1500000), RUN),
    (_uniform(1000003, 2600000), TWO), (_capped(500001, 8), COLD), (_capped(900002, 5), {"k_pull_rows4"} | ONE),
    (_uniform(1000003, 6000000), COLD), (_uniform(6000001, 600000), None), (_uniform(4000037, 20000000), None),
    (pb.rmat(16, 1, 3), RUN), (pb.rmat(22, 1, 3), COLD)])
def test_short_rows_take_the_bins(graph, kernels):
    """Which kernels answer, on both sides of each limit of the rule; the ranks
    against the oracle (L1 <= 1e-6) and against the merge path, which takes any
    graph (each within 1e-6 of the oracle's)."""
    V, s, d = graph
    want, _, _ = RefGraph(V, s, d, True).pagerank(5, 0.85, 0.0)
    with pb.Graph(V, s, d, True) as g:
        hit, (got, st) = _launched(lambda: g.pagerank(5, 0.85, 0.0), KERNELS)
        exits, (again, early) = _launched(lambda: g.pagerank(50, 0.85, 1e-2 * V), KERNELS)
    if kernels == ONE:  # decisions in one launch beat a kernel for each
        assert exits == (RUN if s.size <= 3500000 and V <= 6000000 else ONE)
    with pb.Graph(V, s, d, True, relabel=False) as g:
        plain, (general, _) = _launched(lambda: g.pagerank(5, 0.85, 0.0), KERNELS)
        late, same = g.pagerank(50, 0.85, 1e-2 * V)
    assert plain == {"k_pull_warp"}
    assert kernels is None or hit == kernels
    assert st.iterations == 5 and early.iterations == same.iterations
    assert early.delta == pytest.approx(same.delta, rel=1e-4)
    assert np.abs(got.astype(np.float64) - want / V).sum() <= 1e-6
    assert np.abs(got.astype(np.float64) - general).sum() <= 2e-6
    assert np.abs(again.astype(np.float64) - late).sum() <= 2e-6


HOT = {"k_flat_hot", "k_flat_cold", "k_flat_update"}
ALL_HOT = {"k_flat_hot", "k_flat_update"}


@pytest.mark.parametrize("V,E,long_row,kernels", [
    (300001, 3600000, 0, ALL_HOT), (300001, 3600000, 65, ALL_HOT), (1000003, 16000000, 65, COLD),
    (1000003, 16000000, 400000, COLD), (1376256, 49545216, 0, ALL_HOT), (1376256, 49545215, 65, COLD),
    (1376257, 50000000, 65, COLD), (57344, 4000000, 0, COLD), (57345, 5000000, 100, COLD),
    (300001, 12000000, 9000000, ALL_HOT), (1100003, 15000000, 14000000, HOT), (172032, 774144, 0, RUN)])
def test_streams_follow_the_rows_that_take_part(V, E, long_row, kernels):
    """Hot streams where the rows that take part fill them: not for one long
    row beside short ones, for all rows where the blocks cover the sources and
    a segment has 1.5 edges.  L1 <= 1e-6 of the oracle's ranks."""
    _, s, d = _uniform(V, E)
    d[:long_row] = 7
    want, _, _ = RefGraph(V, s, d, True).pagerank(3, 0.85, 0.0)
    with pb.Graph(V, s, d, True) as g:
        hit, (got, _) = _launched(lambda: g.pagerank(3, 0.85, 0.0), KERNELS)
        again, _ = g.pagerank(3, 0.85, 0.0)
    assert hit == kernels
    assert np.abs(got.astype(np.float64) - want / V).sum() <= 1e-6
    np.testing.assert_array_equal(got, again)


@pytest.mark.parametrize("E", [64000000, 3000000])
def test_small_terms_beside_large_ones(E):
    """Every edge ends in vertex 1, its own among them: a few terms near 0.008
    among millions near 1e-9, which a running 32-bit sum would round away one
    by one.  The oracle's bar (1e-6) on every rank, relatively."""
    import torch

    V = 1000003
    rng = np.random.default_rng(E)
    s, d = rng.integers(0, V, E, dtype=np.uint32), np.ones(E, np.uint32)
    deg = np.maximum(np.bincount(s, minlength=V), 1)
    src, out = torch.as_tensor(s.astype(np.int64)), torch.as_tensor(deg.astype(np.float64))
    x = 1.0 / V / out
    for _ in range(4):
        r = torch.full((V,), 0.15 / V, dtype=torch.float64)
        r[1] += 0.85 * x[src].sum()
        x = r / out
    with pb.Graph(V, s, d, True) as g:
        got, _ = g.pagerank(4, 0.85, 0.0)
    np.testing.assert_allclose(got, r.numpy(), rtol=1e-6, atol=0)


@pytest.mark.parametrize("V,E,share", [(900, 60000, 0.9), (100003, 3000000, 0.9), (300001, 12000000, 0.8),
                                       (100003, 12000000, 0.5)])
def test_infinite_terms_make_infinite_rows(V, E, share):
    """Weights so small that 1 / their sum is infinite: a target's rank is
    infinite, not NaN, whether its row ends in a step or crosses thousands; as
    by the merge path."""
    rng = np.random.default_rng(E)
    s = rng.integers(0, V, E, dtype=np.uint32)
    d = rng.integers(0, V, E, dtype=np.uint32)
    d[rng.random(E) < share] = 1
    w = np.ones(E)
    w[s == 3] = 1e-42
    hit = np.zeros(V, bool)
    hit[d[s == 3]] = True
    assert hit[1]
    for relabel in (False, True):
        with pb.Graph(V, s, d, True, relabel=relabel, weights=w) as g:
            got, _ = g.weighted_pagerank(1, 0.85, 0.0)
        np.testing.assert_array_equal(np.isposinf(got), hit)
        assert np.isfinite(got[~hit]).all()


def _weighted_graph(kind):
    if kind == "hot and cold":
        V, s, d = pb.rmat(20, 12, 7)
    else:
        V, s, d = _uniform(1000003, 9000000)
    return V, s, d, np.random.default_rng(5).uniform(0.1, 10, s.size)


@pytest.mark.parametrize("kind,kernels", [("hot and cold", HOT), ("cold", COLD)])
@pytest.mark.parametrize("early", [False, True])
def test_weights_of_the_cold_stream(kind, kernels, early):
    """Weighted epochs above one launch, with a cold stream: 32-bit ids, their
    weights and padding."""
    V, s, d, w = _weighted_graph(kind)
    eps = 1e-6 * V if early else 0.0
    want, epochs, _ = fp64.weighted_pagerank(V, s, d, w, True, 80 if early else 12, 0.85, eps)
    with pb.Graph(V, s, d, True, weights=w) as g:
        hit, (got, st) = _launched(lambda: g.weighted_pagerank(80 if early else 12, 0.85, eps), KERNELS)
        again, _ = g.weighted_pagerank(80 if early else 12, 0.85, eps)
    assert hit == kernels
    assert abs(st.iterations - epochs) <= (1 if early else 0)
    assert np.abs(got - want).sum() / V <= 1e-6
    np.testing.assert_array_equal(got, again)


@pytest.mark.parametrize("kind", ["hot and cold", "cold"])
def test_not_a_number_beside_cold_edges(kind):
    """A vertex whose out-weights are all 0 gathers as inf, its targets become
    NaN in the first epoch, no other row does."""
    V, s, d, w = _weighted_graph(kind)
    v = int(s[s.size // 2])
    w[s == v] = 0.0
    hit = np.zeros(V, bool)
    hit[d[s == v]] = True
    with pb.Graph(V, s, d, True, weights=w) as g:
        got, _ = g.weighted_pagerank(1, 0.85, 0.0)
    np.testing.assert_array_equal(np.isnan(got), hit)


@pytest.mark.parametrize("scale,ef,kernels", [(10, 24, RUN), (18, 24, COLD), (19, 24, HOT)])
@pytest.mark.parametrize("eps", [0.0, 1e-6])
def test_seed_sets(scale, ef, kernels, eps):
    """Seed-set queries through each form of the flat pull."""
    V, s, d = pb.rmat(scale, ef, 8)
    ref = RefGraph(V, s, d, True)
    seeds = np.random.default_rng(scale).choice(V, 17, replace=False).astype(np.uint32)
    iteration = 100 if eps else 20
    want, epochs, delta = ref.seedset_ppr(seeds, iteration, 0.85, eps)
    with pb.Graph(V, s, d, True) as g:
        hit, (got, st) = _launched(lambda: g.seedset_ppr(seeds, iteration, 0.85, eps), KERNELS)
    assert hit == kernels
    assert abs(st.iterations - epochs) <= (1 if eps else 0)
    # the bar, and one epoch that moves less than eps where one side ends earlier
    assert np.abs(got.astype(np.float64) - want).sum() <= 1e-6 + eps


@pytest.mark.parametrize("name", ["one launch", "separate kernels", "bins", "caller's order"])
@pytest.mark.parametrize("iteration", [1, 2, 3, 4, 5, 9])
def test_epochs_of_an_early_exit(name, iteration):
    """Exits after the first epoch, in the middle and never, around the number of
    epochs that are enqueued ahead: epochs and delta as the oracle's, ranks those
    of as many epochs without an exit."""
    V, s, d = {"one launch": lambda: pb.rmat(13, 16, 2), "separate kernels": lambda: pb.rmat(18, 24, 2),
               "bins": lambda: _capped(1200001, 4), "caller's order": lambda: pb.rmat(13, 16, 2)}[name]()
    ref = RefGraph(V, s, d, True)
    third = ref.pagerank(4, 0.85, 1e-300)[2]
    with pb.Graph(V, s, d, True, relabel=name != "caller's order") as g:
        for eps in (10.0 * V, third * 1.01, 1e-300):
            got, st = g.pagerank(iteration, 0.85, eps)
            want, epochs, dl = ref.pagerank(iteration, 0.85, eps)
            assert st.iterations == epochs
            if epochs > 1:
                assert st.delta == pytest.approx(dl, rel=1e-3)
            assert np.abs(got.astype(np.float64) - want / V).sum() <= 1e-6
            fixed, _ = g.pagerank(epochs, 0.85, 0.0)
            assert np.abs(got.astype(np.float64) - fixed).sum() <= 2e-6


@pytest.mark.parametrize("graph,kernels", [
    (_ring(100003), ONE), (_uniform(1000003, 2600000), RUN), (_uniform(2000003, 5000000), TWO),
    (_uniform(1000003, 3600000), COLD), (_uniform(4000037, 20000000), COLD), (_capped(1200001, 4), ONE)])
def test_short_rows_with_weights(graph, kernels):
    """The same rule with weights, whose limits lie higher; a fixed number of
    epochs and an early exit, against the oracle's bar."""
    V, s, d = graph
    w = np.random.default_rng(V).uniform(0.1, 10, s.size)
    want, _, _ = fp64.weighted_pagerank(V, s, d, w, True, 6, 0.85, 0.0)
    with pb.Graph(V, s, d, True, weights=w) as g:
        hit, (got, _) = _launched(lambda: g.weighted_pagerank(6, 0.85, 0.0), KERNELS)
        early, st = g.weighted_pagerank(6, 0.85, 1e-300)
    assert hit == kernels and 2 <= st.iterations <= 6  # the ring's ranks stand still, to the last bit
    assert np.nansum(np.abs(got - want)) / V <= 1e-6
    assert np.nansum(np.abs(early - want)) / V <= 1e-6
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
