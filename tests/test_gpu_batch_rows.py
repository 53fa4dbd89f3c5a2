"""Rows of the batched pull that many groups and tiles of one CTA share: a hub
whose in-edges end just before, at and after a tile of 2048 merge items, and one
that fills several tiles, among short rows.  Against the FP64 oracle, L1 <= 1e-6
per query as for every 32-bit rank vector; epochs equal."""
import numpy as np
import pytest

import plato_b200 as pb
from oracle import RefGraph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kt", [8, 16, 64])
@pytest.mark.parametrize("hub", [31, 2046, 2047, 2048, 9000])
def test_hub_rows(kt, hub):
    V = 9500
    rng = np.random.default_rng(hub)
    s = np.concatenate([rng.permutation(V)[:hub], rng.integers(0, V, 20000)]).astype(np.uint32)
    d = np.concatenate([np.full(hub, 17), rng.integers(0, V, 20000)]).astype(np.uint32)
    seeds = [[17], [0, 5, 9], [V - 1, 17], [1, 2]]
    ref = RefGraph(V, s, d, True)
    with pb.Graph(V, s, d, True) as g:
        out = g.ppr_batch(seeds, max_iterations=12, eps=0.0, ranks=True, k_tile=kt)
    for q, S in enumerate(seeds):
        want, epochs, _ = ref.seedset_ppr(S, 12, 0.85, 0.0)
        assert out["iterations"][q] == epochs
        assert np.abs(out["ranks"][q].astype(np.float64) - want).sum() <= 1e-6
