"""The deterministic tree around the length at which a list is cut into chunks
(512 arcs), on graphs known to be symmetric and on a caller's CSR."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

bd = pytest.importorskip("beedrill_b200")


def _two_hubs(width):
    """0 - (1..width) - last: the last vertex and 0 have `width` neighbours, ids
    shuffled so that the smallest parent is nowhere in particular in a list."""
    n = width + 2
    rng = np.random.default_rng(width)
    ids = rng.permutation(n)
    mid = np.arange(1, width + 1)
    src = np.concatenate([np.zeros(width, np.int64), mid])
    dst = np.concatenate([mid, np.full(width, n - 1)])
    order = rng.permutation(2 * width)
    return n, ids[src][order], ids[dst][order], int(ids[0])


@pytest.mark.parametrize("width", [1, 31, 32, 33, 511, 512, 513, 1023, 1024, 1025, 5000])
@pytest.mark.parametrize("form", ["edges", "hub", "csr"])
def test_min_parent_around_the_chunk_length(width, form):
    n, src, dst, root = _two_hubs(width)
    g = bd.Graph.from_edges(n, src, dst, bd.ORDER_HUB if form == "hub" else bd.ORDER_INSERTION)
    off, adj = g.csr()
    if form == "csr":
        g = bd.Graph.from_csr(off, adj)
    depth = O.bfs_depth(off, adj, root)
    want = O.min_parent(off, adj, root, depth)
    single = bd.HybridBFS(g, min_parent=True)
    for _ in range(2):
        single.clear()
        single.run(root)
        assert np.array_equal(single.parents(), want)
    ms = bd.BatchedBFS(g, 3, min_parent=True)
    ms.run([root, root, int(src[0])])
    for i, r in enumerate((root, root, int(src[0]))):
        d = O.bfs_depth(off, adj, r)
        assert np.array_equal(ms.depths(i), d)
        assert np.array_equal(ms.parents(i), O.min_parent(off, adj, r, d))


@pytest.mark.parametrize("order", [bd.ORDER_INSERTION, bd.ORDER_HUB])
def test_getters_after_rows_went_to_the_caller(order):
    """run_many_into on a min-parent handle: the getters show the last root."""
    torch = pytest.importorskip("torch")
    g = bd.Graph.rmat(11, 8, seed=3, order=order)
    off, adj = g.csr()
    n = g.num_vertices()
    bfs = bd.HybridBFS(g, min_parent=True)
    roots = [int(r) for r in g.pick_roots(1, 3)]
    bfs.run(roots[2])
    d = torch.empty((2, n), dtype=torch.int32, device="cuda")
    p = torch.empty((2, n), dtype=torch.int64, device="cuda")
    bfs.run_many_into(roots[:2], d.data_ptr(), p.data_ptr())
    depth = O.bfs_depth(off, adj, roots[1])
    assert np.array_equal(d[1].cpu().numpy(), depth)
    assert np.array_equal(bfs.depths(), depth)
    assert O.check(off, adj, roots[1], bfs.parents())


@pytest.mark.parametrize("form", ["edges", "hub", "csr"])
def test_getters_and_rows_hold_the_same_tree(form):
    """run_many_into on a min-parent handle leaves the smallest parents to the
    getters too, whatever kind of run came before or comes next."""
    torch = pytest.importorskip("torch")
    g = bd.Graph.rmat(12, 16, seed=7, order=bd.ORDER_HUB if form == "hub" else bd.ORDER_INSERTION)
    off, adj = g.csr()
    if form == "csr":
        g = bd.Graph.from_csr(off, adj)
    n = g.num_vertices()
    bfs = bd.HybridBFS(g, min_parent=True)
    roots = [int(r) for r in g.pick_roots(1, 4)]
    want = [O.min_parent(off, adj, r, O.bfs_depth(off, adj, r)) for r in roots]
    d = torch.empty((2, n), dtype=torch.int32, device="cuda")
    p = torch.empty((2, n), dtype=torch.int64, device="cuda")
    for k in (0, 2):
        bfs.run_many_into(roots[k:k + 2], d.data_ptr(), p.data_ptr())
        assert np.array_equal(p.cpu().numpy(), want[k:k + 2])
        for _ in range(2):
            assert np.array_equal(bfs.parents(), want[k + 1])
        assert bfs.check(roots[k + 1])
        bfs.run(roots[k])
        assert np.array_equal(bfs.parents(), want[k])
    bfs.run_many(roots)
    assert np.array_equal(bfs.parents(), want[3])


def test_new_handles_beside_work_on_the_default_stream():
    """A handle made and used while the default stream is busy, which handles'
    streams do not wait for: its counters are clear before its first launch, and
    nothing of its making is left to come after it."""
    torch = pytest.importorskip("torch")
    n, src, dst, root = _two_hubs(5000)
    g = bd.Graph.from_edges(n, src, dst)
    off, adj = g.csr()
    want = O.min_parent(off, adj, root, O.bfs_depth(off, adj, root))
    for make in (lambda: bd.HybridBFS(g, min_parent=True), lambda: bd.BatchedBFS(g, 2, min_parent=True)):
        torch.cuda._sleep(1 << 28)  # some 0.15 s
        handle = make()
        parents = handle.parents if isinstance(handle, bd.HybridBFS) else lambda: handle.parents(0)
        for _ in range(2):
            handle.run(root if isinstance(handle, bd.HybridBFS) else [root, root])
            assert np.array_equal(parents(), want)
            torch.cuda.synchronize()
