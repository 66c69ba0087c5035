"""Batch.bfs_multi hands the C call one source address and one count per graph,
whatever form the lists have; list counts that do not match are refused before
it. The C call is replaced by one that records what it was given."""
import ctypes
from types import SimpleNamespace

import numpy as np
import pytest

import gpma_bfs_gb300 as G


@pytest.fixture
def calls(monkeypatch):
    """The source lists of every C call made, as C reads them."""
    seen = []

    def gpma_batch_bfs_multi(batch, graphs, srcs, nsrc, k, levels, reached, stream):
        addr = (ctypes.c_uint64 * k).from_address(srcs)
        count = (ctypes.c_uint32 * k).from_address(nsrc)
        seen.append([list((ctypes.c_uint32 * count[i]).from_address(addr[i])) for i in range(k)])
        return 0

    monkeypatch.setattr(G, "lib", lambda: SimpleNamespace(gpma_batch_bfs_multi=gpma_batch_bfs_multi))
    return seen


def _batch_and_graphs(k):
    b = G.Batch.__new__(G.Batch)
    b._h = None
    return b, [SimpleNamespace(handle=ctypes.c_void_p(16 * (i + 1)), row_num=9) for i in range(k)]


@pytest.mark.parametrize("graphs, lists", [(3, 1), (3, 2), (1, 0), (1, 2), (2, 5), (0, 1)])
def test_list_count_must_match(monkeypatch, graphs, lists):
    made = []
    monkeypatch.setattr(G, "lib", lambda: SimpleNamespace(gpma_batch_bfs_multi=lambda *a: made.append(a) or 0))
    b, gs = _batch_and_graphs(graphs)
    for levels in (False, True):
        with pytest.raises(ValueError):
            b.bfs_multi(gs, [[1, 2]] * lists, levels=levels)
    assert not made


@pytest.mark.parametrize("form, want", [
    ([[1], [2, 3]], [[1], [2, 3]]),
    ([4, [5]], [[4], [5]]),  # a single node in place of a list
    ([np.uint32(7), np.array(8)], [[7], [8]]),
    (np.array([[1, 2], [3, 4]]), [[1, 2], [3, 4]]),
    ((np.arange(6, dtype=np.int64)[::2], (5,)), [[0, 2, 4], [5]]),
])
def test_source_forms(calls, form, want):
    b, gs = _batch_and_graphs(2)
    _, parts = b.bfs_multi(gs, form)
    assert calls == [want]
    assert [len(p) for p in parts] == [len(w) for w in want]
