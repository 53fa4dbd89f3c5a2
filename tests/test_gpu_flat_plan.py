"""The flat pull's reports and plans at the edges of what takes it: the delta
of a call whose only pull epoch is the final one, and graphs whose rows,
sources or memory do not suit a flat plan."""
import numpy as np
import pytest

import plato_b200 as pb
from oracle import RefGraph

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
