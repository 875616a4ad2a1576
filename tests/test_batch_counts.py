"""counts() of a batched handle after a run that failed: the library's last run may
then have more or fewer roots than the last one the Python object saw succeed."""
import types

import numpy as np
import pytest

import beedrill_b200 as bd


class _Lib:
    """The two calls that counts() makes, for a handle whose last run had `roots`."""

    def __init__(self, roots):
        self.roots = roots

    def bd_msbfs_count_traversed_edges(self, handle, i, edges, reached):
        return bd.BD_OK if 0 <= i < self.roots else -7

    def bd_msbfs_counts(self, handle, edges, reached):
        for out in (edges, reached):
            assert len(out) >= self.roots, "the library writes past the array"
            out[:self.roots] = 100 + np.arange(self.roots)
        return bd.BD_OK


@pytest.mark.parametrize("seen,roots,max_roots", [(5, 5, 5), (5, 5, 64), (3, 64, 64), (64, 64, 130)])
def test_counts_fit_the_library_s_last_run(monkeypatch, seen, roots, max_roots):
    fake = _Lib(roots)
    monkeypatch.setattr(bd, "lib", lambda: fake)
    monkeypatch.setattr(bd, "_ptr", lambda a, ct: a)
    ms = types.SimpleNamespace(_h=None, count=seen, max_roots=max_roots)
    m, n = bd.BatchedBFS.counts(ms)
    assert m.tolist() == n.tolist() == list(range(100, 100 + seen))


def test_counts_of_fewer_roots_are_an_error(monkeypatch):
    fake = _Lib(2)
    monkeypatch.setattr(bd, "lib", lambda: fake)
    monkeypatch.setattr(bd, "_ptr", lambda a, ct: a)
    with pytest.raises(bd.BeedrillError):
        bd.BatchedBFS.counts(types.SimpleNamespace(_h=None, count=5, max_roots=64))
