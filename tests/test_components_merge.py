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
