"""HyperLogLog epochs on rows whose number of sources lies at the limits of
their work shares: a staged round of 32 ids, a team's and a warp's share, a
CTA's; in both directions, on vertex counts around a chunk and on both sides
of the wide team share (2^18 vertices).  Registers and degrees equal the
oracle's bit for bit."""
import numpy as np
import pytest

import plato_b200 as pb
from oracle import hll

pytestmark = pytest.mark.gpu

DEGREES = [1, 7, 8, 31, 32, 33, 63, 64, 65, 127, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 2047, 2048, 2049, 5000]


def _graph(V, seed):
    """Rows with the listed in-degrees among light ones, and as many vertices with those out-degrees."""
    rng = np.random.default_rng(seed)
    rows = rng.choice(V, 2 * len(DEGREES), replace=False)
    s, d = [rng.integers(0, V, V)], [rng.integers(0, V, V)]
    for row, n in zip(rows, DEGREES + DEGREES):
        s.append(rng.integers(0, V, n))
        d.append(np.full(n, row))
    for row, n in zip(rows[::-1], DEGREES):
        s.append(np.full(n, row))
        d.append(rng.integers(0, V, n))
    return np.concatenate(s).astype(np.uint32), np.concatenate(d).astype(np.uint32)


@pytest.mark.parametrize("bits", [4, 5, 6, 7, 8, 9, 10, 12])
@pytest.mark.parametrize("relabel", [True, False])
def test_registers(bits, relabel):
    V = 6001 + bits
    s, d = _graph(V, bits)
    _, anfs_want, want, modes = hll.hyperanf(V, s, d, True, bits=bits, iterations=3, push_threshold=0.0)
    with pb.Graph(V, s, d, True, relabel=relabel) as g:
        _, anfs, got, st = g.hyperanf(3, bits, push_threshold=0.0, registers=True)
    np.testing.assert_array_equal(got, want)
    np.testing.assert_allclose(anfs, anfs_want, rtol=1e-12)
    assert [m == "push" for m in st.mode_trace] == modes


@pytest.mark.parametrize("V", [262143, 262145])
def test_registers_of_many_rows(V):
    s, d = _graph(V, 3)
    want = hll.hyperanf(V, s, d, True, bits=5, iterations=2, push_threshold=0.0)[2]
    with pb.Graph(V, s, d, True) as g:
        got = g.hyperanf(2, 5, push_threshold=0.0, registers=True)[2]
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("bits", [4, 6, 9])
def test_degrees_of_targets(bits):
    V = 5003
    s, d = _graph(V, 20 + bits)
    targets = np.random.default_rng(bits).random(V) < 0.3
    for push in (0.0, 0.05):
        want = hll.nstep_degrees(V, s, d, True, step=2, bits=bits, kind="both", is_directed=True, targets=targets,
                                 push_threshold=push)
        with pb.Graph(V, s, d, True) as g:
            din, dout, _ = g.nstep_degrees(2, bits, "both", True, targets, push)
        np.testing.assert_array_equal(din, want[0])
        np.testing.assert_array_equal(dout, want[1])
