"""Parts of chunks: however few chunks a frontier has and however long a chunk is
(the chunk_edges option), the parts that the warps take cover every arc once."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
#include "bd_split.h"
extern "C" int cut_of(long long chunks, unsigned chunk, long long nw)
{
    return bd::dev::split_chunks(chunks, chunk, nw);
}
extern "C" long long check_polls(long long degree) { return bd::dev::check_polls(degree); }
extern "C" int long_chunk(int arcs) { return bd::dev::long_chunk(arcs); }
extern "C" long long part_of(unsigned chunk, int cut) { return bd::dev::split_part(chunk, cut); }
"""


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    d = tmp_path_factory.mktemp("split")
    (d / "split.cc").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "beedrill_b200", "csrc"), "-o", str(d / "split.so"),
                    str(d / "split.cc")], check=True)
    so = ctypes.CDLL(str(d / "split.so"))
    so.cut_of.argtypes = [ctypes.c_longlong, ctypes.c_uint, ctypes.c_longlong]
    so.check_polls.argtypes, so.check_polls.restype = [ctypes.c_longlong], ctypes.c_longlong
    so.part_of.argtypes, so.part_of.restype = [ctypes.c_uint, ctypes.c_int], ctypes.c_longlong
    return so


def test_parts_cover_their_chunk(split):
    for chunk in [*range(1, 4097), 2**20 - 1, 2**20 + 1, 2**31 - 33, 2**31 - 1]:
        for cut in range(split.cut_of(1, chunk, 1 << 40) + 1):
            part = split.part_of(chunk, cut)
            assert part % 32 == 0 and part << cut >= chunk, (chunk, cut, part)


def test_chunks_of_long_lists_for_any_heavy_degree(split):
    for arcs in (1, 63, 64, 65, 1023, 1024, 1025, 4096, 2**30 - 1, 2**30, 2**31 - 1):
        assert split.long_chunk(arcs) == min(2048, max(128, 2 * arcs)), arcs


def test_the_check_waits_for_the_longest_list(split):
    # 32 lists of 128 arcs in three polls each
    for degree in (0, 1, 1 << 20, 1 << 28, 1 << 32, 1 << 34):
        assert split.check_polls(degree) >= max(4000000, 32 * 3 * degree // 128)


def _star(leaves):
    """A hub with `leaves` neighbours, the last of which are the ends of tails."""
    n = leaves + 1 + 40
    src = np.concatenate([np.zeros(leaves, np.int64), np.arange(leaves - 39, leaves + 1)])
    dst = np.concatenate([np.arange(1, leaves + 1), np.arange(leaves + 1, n)])
    return n, src, dst


@pytest.mark.gpu
@pytest.mark.parametrize("chunk_edges", [1, 33, 65, 129, 193, 257, 260, 263, 1027])
@pytest.mark.parametrize("form", ["star", "rmat"])
def test_searches_with_any_chunk_length(chunk_edges, form):
    bd = pytest.importorskip("beedrill_b200")
    from oracle import oracle as O

    if form == "star":
        g = bd.Graph.from_edges(*_star(9001))
        roots = [0, 1, g.num_vertices() - 1]
    else:
        g = bd.Graph.rmat(13, 16, seed=chunk_edges)
        roots = [int(r) for r in g.pick_roots(chunk_edges, 3)]
    off, adj = g.csr()
    want = [O.bfs_depth(off, adj, r) for r in roots]
    single = bd.HybridBFS(g, alg="top_down", chunk_edges=chunk_edges)
    for r, d in zip(roots, want):
        single.run(r)
        assert np.array_equal(single.depths(), d)
        assert O.check(off, adj, r, single.parents())
    for k in (1, 3):  # a batch of one has the fewest chunks in a level
        ms = bd.BatchedBFS(g, k, chunk_edges=chunk_edges, force_dir=0)
        ms.run(roots[:k])
        for i in range(k):
            assert np.array_equal(ms.depths(i), want[i])
            assert O.check(off, adj, roots[i], ms.parents(i))
