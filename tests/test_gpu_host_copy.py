"""Result vectors reach pageable host memory whole: sizes around the limit of
the plain copy (1 MB), a chunk (256 KB) and a half (4 MB) of the staging
memory, several rounds of it, and several graphs at once from threads.  The
expected vectors come through a caller's pinned buffer or device memory,
byte for byte."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

import plato_b200 as pb
from plato_b200 import _lib

pytestmark = pytest.mark.gpu


def _graph(V):
    rng = np.random.default_rng(V)
    s = rng.integers(0, V, 2 * V, dtype=np.uint32)
    d = rng.integers(0, V, 2 * V, dtype=np.uint32)
    return s, d, pb.Graph(V, s, d, True)


@pytest.mark.parametrize("V", [262143, 262144, 327681, 1048576, 1048577, 2097153, 3211265])
def test_every_byte_arrives(V):
    s, d, g = _graph(V)
    with g:
        want = torch.empty(V, device="cuda")
        g.pagerank_device(want.data_ptr(), 3)
        torch.cuda.synchronize()
        want = want.cpu().numpy()
        for _ in range(2):
            np.testing.assert_array_equal(g.pagerank(3)[0], want)
        pinned = torch.empty(V, pin_memory=True)
        o = _lib.PagerankOpts(3, 0.85, 0.0)
        _lib.check(_lib.load().plato_pagerank(g.handle, C.byref(o), C.c_void_p(pinned.data_ptr()), None), "pagerank")
        np.testing.assert_array_equal(pinned.numpy(), want)
        np.testing.assert_array_equal(g.out_degrees(), np.bincount(s, minlength=V).astype(np.uint32))
        lev, par, _ = g.bfs(int(s[0]))
        reached = np.flatnonzero((lev != pb.PLATO_LEVEL_UNREACHED) & (lev > 0))
        assert lev[s[0]] == 0 and par[s[0]] == s[0]
        assert (lev[par[reached]] + 1 == lev[reached]).all()
        assert (par[lev == pb.PLATO_LEVEL_UNREACHED] == V).all()


def test_graphs_on_several_threads():
    graphs = [_graph(1200001 + k) for k in range(4)]
    want = [g.pagerank(2)[0] for _, _, g in graphs]
    wrong = []

    def work(k):
        for _ in range(5):
            if not np.array_equal(graphs[k][2].pagerank(2)[0], want[k]):
                wrong.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for _, _, g in graphs:
        g.close()
    assert not wrong
