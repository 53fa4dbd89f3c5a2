"""The flat pull's reports and plans at the edges of what takes it: the delta
of a call whose only pull epoch is the final one, and graphs whose rows,
sources or memory do not suit a flat plan."""
import numpy as np
import pytest

import plato_b200 as pb
from oracle import RefGraph
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
