"""The device check around the list lengths at which it changes who looks through
a list (16 and 2048 arcs) or splits it (1024), on symmetric graphs and on a
caller's CSR, with a tree that is right and with one mistake."""
import time

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

bd = pytest.importorskip("beedrill_b200")


@pytest.mark.parametrize("width", [2, 15, 16, 17, 18, 1023, 1024, 1025, 2047, 2048, 2049, 2050, 9000])
@pytest.mark.parametrize("form", ["edges", "csr"])
def test_long_lists(width, form):
    """root - (width vertices) - last, but one of the middle is not tied to last."""
    n = width + 2
    rng = np.random.default_rng(width)
    ids = rng.permutation(n)
    mid, odd = ids[1:-1], int(ids[1])
    src = np.concatenate([np.full(width, ids[0]), mid[1:]])
    dst = np.concatenate([mid, np.full(width - 1, ids[-1])])
    order = rng.permutation(len(src))
    g = bd.Graph.from_edges(n, src[order], dst[order])
    off, adj = g.csr()
    if form == "csr":
        g = bd.Graph.from_csr(off, adj)
    root, last = int(ids[0]), int(ids[-1])
    depth = O.bfs_depth(off, adj, root)
    right = O.min_parent(off, adj, root, depth)
    right[root] = root
    assert O.check(off, adj, root, right)
    assert g.check_parents(root, right) == (True, -1)
    for v, p in ((last, odd), (last, root), (odd, last), (root, odd), (int(mid[-1]), odd)):
        wrong = right.copy()
        wrong[v] = p
        assert not O.check(off, adj, root, wrong)
        assert g.check_parents(root, wrong) == (False, v)
    bfs = bd.HybridBFS(g)
    for r in (root, last, odd):
        bfs.run(r)
        assert bfs.check(r) and bfs.check(r)


def test_a_small_graph_takes_no_longer_than_a_large_one():
    """A frontier of a few vertices with lists of hundreds of arcs is dealt to many
    warps: as one warp's work it made the check of a scale-14 graph three times as
    long as that of a graph 16 times its size (the bound allows 1.5 times)."""
    best = {}
    for scale in (14, 18):
        g = bd.Graph.rmat(scale, 16, seed=scale, order=bd.ORDER_HUB)
        root = int(g.pick_roots(3, 8)[7])
        bfs = bd.HybridBFS(g)
        bfs.run(root)
        times = []
        for _ in range(16):
            t0 = time.perf_counter()
            assert bfs.check(root)
            times.append(time.perf_counter() - t0)
        best[scale] = min(times)
    assert best[14] < 1.5 * best[18], best
