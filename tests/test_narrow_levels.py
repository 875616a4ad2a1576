"""Levels that one CTA runs alone: frontiers around the bounds of its queue
(5/8 of a block of vertices, 5 blocks of arcs), runs of more levels than it
takes in one go, many sources, and graphs small enough for its bottom-up steps."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

bd = pytest.importorskip("beedrill_b200")


def _graph(n, edges, order=bd.ORDER_INSERTION):
    src, dst = np.array(edges, np.int64).reshape(-1, 2).T
    return bd.Graph.from_edges(n, src, dst, order)


def _broom(width, leaves):
    """Root 0 -> `width` vertices -> `leaves` leaves each -> one last vertex."""
    mid = list(range(1, 1 + width))
    edges = [(0, v) for v in mid]
    nxt = 1 + width
    last = nxt + width * leaves
    for v in mid:
        for _ in range(leaves):
            edges += [(v, nxt), (nxt, last)]
            nxt += 1
    return last + 1, edges


def _verify(bfs, g, root):
    off, adj = g.csr()
    depth = O.bfs_depth(off, adj, root)
    assert np.array_equal(bfs.depths(), depth)
    parent = bfs.parents()
    assert O.check(off, adj, root, parent)
    assert bfs.count_num_traversed_edges() == O.count_traversed(off, parent)
    return off, depth


@pytest.mark.parametrize("block", [256, 512, 1024])
@pytest.mark.parametrize("width,leaves", [(1, 1), (1, 3000), (159, 2), (160, 7), (161, 8), (319, 3),
                                          (320, 7), (321, 1), (640, 3), (641, 8), (1700, 2)])
def test_frontiers_at_the_bounds(block, width, leaves):
    n, edges = _broom(width, leaves)
    g = _graph(n, edges)
    for alg in ("top_down", "beamer_hybrid", "bottom_up"):
        bfs = bd.HybridBFS(g, alg=alg, block_size=block)
        for root in (0, n - 1, 1):
            bfs.run(root)
            off, depth = _verify(bfs, g, root)
            if alg == "beamer_hybrid":
                dirs, found = O.beamer_sequence(off, depth, root, g.num_edges())
                assert bfs.directions() == dirs
                assert [s["found"] for s in bfs.steps()] == found.tolist()


@pytest.mark.parametrize("length", [2, 127, 128, 129, 130, 1000])
def test_long_runs_of_narrow_levels(length):
    g = bd.Graph.grid(1, length, 0.0, 0)
    for alg in ("top_down", "beamer_hybrid"):
        bfs = bd.HybridBFS(g, alg=alg)
        bfs.run(0)
        _verify(bfs, g, 0)
        assert len(bfs.steps()) == length
        assert all(s["ns"] >= 0 for s in bfs.steps())


@pytest.mark.parametrize("order", [bd.ORDER_INSERTION, bd.ORDER_HUB])
@pytest.mark.parametrize("count", [1, 2, 31, 320, 321, 1500])
def test_many_sources(order, count):
    """Sources past the shared queue, repeated ones and ones without edges."""
    g = bd.Graph.rmat(12, 8, seed=count, order=order)
    off, adj = g.csr()
    n = g.num_vertices()
    rng = np.random.default_rng(count)
    src = rng.integers(0, n, count)
    src[count // 2] = src[0]
    src[-1] = int(np.flatnonzero(np.diff(off) == 0)[0])
    bfs = bd.HybridBFS(g)
    st = bfs.run_multi(src)
    want = np.full(n, -1, np.int64)
    for s in np.unique(src):
        d = O.bfs_depth(off, adj, int(s))
        want = np.where((d >= 0) & ((want < 0) | (d < want)), d, want)
    assert np.array_equal(bfs.depths(), want)
    assert st.reached == int((want >= 0).sum())
    parent = bfs.parents()
    reached = want > 0
    assert np.array_equal(want[parent[reached]], want[reached] - 1)
    assert np.array_equal(parent[want == 0], np.flatnonzero(want == 0))


def test_long_source_lists_under_a_short_wait_bound():
    """spin_limit bounds the wait for one level.  CTA 0 needs several times as long
    for the sources (2048 rounds of some 3 us, against 2000 polls of about 0.7 us);
    the levels themselves, and the whole call before sources were set up by the one
    launch, stay far below it."""
    g = bd.Graph.rmat(20, 8, seed=1)
    n = g.num_vertices()
    bfs = bd.HybridBFS(g, spin_limit=2000)
    assert bfs.run_multi(np.arange(n)).reached == n
    assert not bfs.depths().any()
    assert np.array_equal(bfs.parents(), np.arange(n))


@pytest.mark.parametrize("scale", [8, 11, 12, 13])
def test_small_graphs_bottom_up(scale):
    g = bd.Graph.rmat(scale, 6, seed=scale)
    for alg in ("bottom_up", "beamer_hybrid"):
        for block in (256, 1024):
            bfs = bd.HybridBFS(g, alg=alg, block_size=block)
            for root in g.pick_roots(scale, 3):
                bfs.run(int(root))
                _verify(bfs, g, int(root))


@pytest.mark.parametrize("order", [bd.ORDER_INSERTION, bd.ORDER_HUB])
@pytest.mark.parametrize("scale,factor", [(9, 30), (10, 30), (11, 4), (12, 4), (12, 16), (13, 2)])
def test_small_graphs_bottom_up_in_either_layout(scale, factor, order):
    """Graphs on both sides of the sizes and arc counts up to which one CTA takes a
    bottom-up level, which depend on the numbering."""
    g = bd.Graph.rmat(scale, factor, seed=scale + factor, order=order)
    for block in (256, 512):
        for alg in ("bottom_up", "beamer_hybrid"):
            bfs = bd.HybridBFS(g, alg=alg, block_size=block)
            for root in g.pick_roots(scale, 3):
                bfs.run(int(root))
                _verify(bfs, g, int(root))
