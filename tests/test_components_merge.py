"""Components whose trees have to be merged in more than one round: pieces of
ragged sizes (some of one vertex), two large ones of equal size, and ids in an
order that makes the smallest id of a piece far from its hubs."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

bd = pytest.importorskip("beedrill_b200")


@pytest.mark.parametrize("pieces", [[1], [2, 1], [31, 32, 33], [1023, 1, 1025, 7], [40, 3000, 3000, 2, 2],
                                    [20000, 20000, 500, 1, 1, 90]])
@pytest.mark.parametrize("form", ["tree", "dense", "path"])
def test_ragged_pieces(pieces, form):
    rng = np.random.default_rng(len(pieces) * 7 + pieces[0])
    n = sum(pieces)
    src, dst, base = [], [], 0
    for k in pieces:
        v = np.arange(1, k)
        if form == "path":
            up = v - 1
        else:
            up = (rng.random(k - 1) * v).astype(np.int64)
        src.append(base + v)
        dst.append(base + up)
        if form == "dense" and k > 3:
            e = rng.integers(0, k, (2, 6 * k))
            e = e[:, e[0] != e[1]]
            src.append(base + e[0])
            dst.append(base + e[1])
        base += k
    ids = rng.permutation(n)
    src, dst = ids[np.concatenate(src)], ids[np.concatenate(dst)]
    order = rng.permutation(len(src))
    for how in (bd.ORDER_INSERTION, bd.ORDER_SORTED, bd.ORDER_HUB):
        g = bd.Graph.from_edges(n, src[order], dst[order], how)
        off, adj = g.csr()
        labels, sizes, count, _ = O.components(off, adj)
        c = bd.Components(g)
        for _ in range(2):
            assert c.run().num_components == count
        assert np.array_equal(c.labels(), labels)
        assert np.array_equal(c.sizes(), sizes)
        assert c.check()


def _comb(spine, teeth):
    """A path of `spine` vertices, a path of `teeth` more hanging from each."""
    v = np.arange(spine - 1)
    src, dst, prev = [v], [v + 1], np.arange(spine)
    for k in range(1, teeth + 1):
        cur = k * spine + np.arange(spine)
        src.append(prev)
        dst.append(cur)
        prev = cur
    return spine * (teeth + 1), np.concatenate(src), np.concatenate(dst)


def test_ids_along_a_path_take_no_longer_than_shuffled_ones():
    """Chains of parents as long as the graph is deep, which hooking makes of ids
    that follow a path, are crossed in steps that double.  Walked arc by arc they
    made this comb three times as slow as the same one with shuffled ids."""
    n, src, dst = _comb(100000, 3)
    ids = np.random.default_rng(0).permutation(n)
    best = []
    for s, d in ((src, dst), (ids[src], ids[dst])):
        c = bd.Components(bd.Graph.from_edges(n, s, d))
        assert c.run().num_components == 1
        best.append(min(c.run().ms for _ in range(9)))
    assert best[0] < 1.5 * best[1], best


@pytest.mark.parametrize("n", [5 * 148 * 2048 + d for d in (-257, -1, 0, 1, 255, 256, 257)])
def test_chains_around_the_flattening_s_border(n):
    """Ids along two paths with an isolated vertex between, at sizes around the one
    from which a thread points two vertices at their roots."""
    half = n // 2
    v = np.concatenate([np.arange(half - 1), np.arange(half + 1, n - 1)])
    c = bd.Components(bd.Graph.from_edges(n, v, v + 1))
    for _ in range(2):
        assert c.run().num_components == 3
    want = np.zeros(n, np.int64)
    want[half:] = half + 1
    want[half] = half
    assert np.array_equal(c.labels(), want)
    sizes = c.sizes()
    assert (sizes[0], sizes[half], sizes[half + 1]) == (half, 1, n - half - 1)


@pytest.mark.parametrize("degree", [1, 2, 31, 33, 4096, 4097])
def test_walk_over_lists_of_one_length(degree):
    """No large tree: stars and pairs side by side, so that every list is walked,
    those of the hubs at lengths around a warp's round and the heavy pass."""
    stars = 3 if degree > 100 else 400
    base = np.arange(stars) * (degree + 1)
    src = np.repeat(base, degree)
    dst = src + np.tile(np.arange(1, degree + 1), stars)
    n = stars * (degree + 1)
    ids = np.random.default_rng(degree).permutation(n)
    for form in ("edges", "csr"):
        g = bd.Graph.from_edges(n, ids[src], ids[dst])
        off, adj = g.csr()
        if form == "csr":
            g = bd.Graph.from_csr(off, adj)
        labels, sizes, count, _ = O.components(off, adj)
        c = bd.Components(g)
        assert c.run().num_components == count == stars
        assert np.array_equal(c.labels(), labels)
        assert np.array_equal(c.sizes(), sizes)
