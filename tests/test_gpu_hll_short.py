"""HyperLogLog epochs on graphs without a long row, whose chunks of rows go to the
warps by number first: vertex counts around a chunk, around what one pass over
the warps covers and past it, at every width that takes the way, and one row
more than it allows.  Registers equal the oracle's bit for bit."""
import numpy as np
import pytest

import plato_b200 as pb
from oracle import hll

pytestmark = pytest.mark.gpu


def _graph(V, k, seed, long_row=0):
    rng = np.random.default_rng(seed)
    d = np.repeat(np.arange(V), k)
    s = rng.integers(0, V, d.size)
    s, d = np.append(s, rng.integers(0, V, long_row)), np.append(d, np.full(long_row, V // 2))
    return s.astype(np.uint32), d.astype(np.uint32)


@pytest.mark.parametrize("bits", [4, 5, 6, 7, 8, 9])
@pytest.mark.parametrize("V", [1, 3, 33, 4737, 37889, 75777])
def test_registers(bits, V):
    s, d = _graph(V, 2, V + bits)
    _, anfs_want, want, _ = hll.hyperanf(V, s, d, True, bits=bits, iterations=3, push_threshold=0.0)
    with pb.Graph(V, s, d, True) as g:
        _, anfs, got, _ = g.hyperanf(3, bits, push_threshold=0.0, registers=True)
    np.testing.assert_array_equal(got, want)
    np.testing.assert_allclose(anfs, anfs_want, rtol=1e-12)


@pytest.mark.parametrize("bits,V,long_row", [(4, 300007, 0), (6, 300007, 0), (6, 20011, 62), (6, 20011, 63),
                                             (6, 300007, 255), (9, 50021, 600)])
def test_registers_past_one_pass_and_beside_a_long_row(bits, V, long_row):
    s, d = _graph(V, 2, bits, long_row)
    want = hll.hyperanf(V, s, d, True, bits=bits, iterations=2, push_threshold=0.0)[2]
    with pb.Graph(V, s, d, True) as g:
        got = g.hyperanf(2, bits, push_threshold=0.0, registers=True)[2]
    np.testing.assert_array_equal(got, want)
