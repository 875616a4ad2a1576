"""The device check around the list lengths at which it changes who looks through
a list (16 and 2048 arcs) or splits it (1024), on symmetric graphs and on a
caller's CSR, with a tree that is right and with one mistake."""
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
