"""Result rows at the sizes where the kernel that writes them changes (37,888 and
227,328 vertices), with an odd number of vertices, and with roots so far apart
that vertices run out of delivery records."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

bd = pytest.importorskip("beedrill_b200")


@pytest.mark.parametrize("rows,cols", [(1, 5), (37, 1023), (37, 1024), (64, 592), (222, 1024), (223, 1023),
                                       (222, 1023), (223, 1024)])
@pytest.mark.parametrize("order", [bd.ORDER_INSERTION, bd.ORDER_HUB])
@pytest.mark.parametrize("roots", [3, 64, 71])
def test_rows_around_the_variants(rows, cols, order, roots):
    g = bd.Graph.grid(rows, cols, 0.01, rows, order=order)
    off, adj = g.csr()
    n = g.num_vertices()
    src = np.random.default_rng(n).integers(0, n, roots)
    ms = bd.BatchedBFS(g, roots, materialize=True)
    ms.run(src)
    for i in range(0, roots, max(1, roots // 5)):
        depth = O.bfs_depth(off, adj, int(src[i]))
        assert np.array_equal(ms.depths(i), depth)
        parent = ms.parents(i)
        assert O.check(off, adj, int(src[i]), parent)
        deg = np.diff(off)
        unreached = depth < 0
        assert np.array_equal(parent[unreached], np.where(deg[unreached] > 0, -deg[unreached], -1))
