"""Setup and per-lane counts of a batch: groups of 1 to 64 lanes, many equal
roots, and roots spread over many components (every component then holds
another set of lanes, the case the counting kernel cannot take in one go)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

bd = pytest.importorskip("beedrill_b200")


def _pieces():
    """Components of ragged sizes (1 x k grids and one RMAT graph) in one CSR."""
    parts = [bd.Graph.grid(1, 1 + (7 * i) % 45, 0.0, i) for i in range(50)]
    parts.append(bd.Graph.rmat(9, 8, seed=9))
    g, base = bd.Graph.concat(parts)
    return g, base


@pytest.mark.parametrize("lanes", [1, 2, 31, 32, 33, 63, 64, 65, 129])
@pytest.mark.parametrize("spread", ["components", "equal", "pairs"])
def test_counts_of_every_lane(lanes, spread):
    g, base = _pieces()
    off, adj = g.csr()
    if spread == "components":
        roots = [int(base[(3 * i) % 51]) for i in range(lanes)]
    elif spread == "equal":
        roots = [int(base[50]) + 5] * lanes
    else:
        roots = [int(base[50]) + (i // 2) % 40 for i in range(lanes)]
    ms = bd.BatchedBFS(g, lanes, materialize=True)
    for _ in range(2):
        ms.run(roots)
    m_c, n_c = ms.counts()
    for i in range(0, lanes, max(1, lanes // 9)):
        depth = O.bfs_depth(off, adj, roots[i])
        assert np.array_equal(ms.depths(i), depth)
        parent = ms.parents(i)
        assert O.check(off, adj, roots[i], parent)
        assert m_c[i] == O.count_traversed(off, parent)
        assert n_c[i] == int((depth >= 0).sum())
