"""BFS of an array large enough for the long work items (2^27 slots and more):
short rows, words of many rows, rows of several items, against a BFS of the edge
list, and against the multi-source kernel and the whole-array sweep."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_long_items_equal_edge_list_bfs(built_lib):
    import gpma_bfs_gb300 as G
    rng = np.random.default_rng(5)
    rows = 72_000_000  # the guards alone fill 2^27 slots
    core = 60_000
    src = np.concatenate([rng.integers(0, core, 600_000), np.full(3000, 7), np.full(513, 40_001),
                          rng.integers(0, rows, 200_000), np.arange(core, core + 64).repeat(20)])
    dst = np.concatenate([rng.integers(0, core, 600_000), rng.integers(0, rows, 3000), rng.integers(0, rows, 513),
                          rng.integers(0, rows, 200_000), rng.integers(0, rows, 64 * 20)])
    keep = src != dst
    keys = np.unique((src[keep].astype(np.uint64) << np.uint64(32)) | dst[keep].astype(np.uint64))
    g = G.GPMA(rows)
    G.update_gpma(g, keys, np.ones(len(keys), np.uint8))
    assert g.geometry()["size"] >= 1 << 27
    s, d = (keys >> np.uint64(32)).astype(np.int64), (keys & np.uint64(0xFFFFFFFF)).astype(np.int64)
    first = np.searchsorted(s, np.arange(rows + 1))
    want = np.zeros(rows, np.uint32)
    front, level = np.array([7]), 1
    while len(front):
        want[front] = level
        n = first[front + 1] - first[front]
        at = np.repeat(first[front] - np.cumsum(n) + n, n) + np.arange(n.sum())
        front = np.unique(d[at])
        front, level = front[want[front] == 0], level + 1
    got, reached = G.gpma_bfs(g, rows, 0, 7)
    assert np.array_equal(got, want) and reached == np.count_nonzero(want)
    before = G.get_tuning()["bfs_dense_div"]
    try:
        G.set_tuning(bfs_dense_div=1000000)
        assert np.array_equal(G.gpma_bfs(g, rows, 0, 7)[0], want)
    finally:
        G.set_tuning(bfs_dense_div=before)
    assert np.array_equal(G.gpma_bfs_multi(g, [7])[0][0], want)
    g.close()
