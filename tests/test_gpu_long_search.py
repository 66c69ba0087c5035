"""Searches of 40,000 levels: the grid barrier's counter starts over in the middle
of the launch (after 65,536 rounds; a level takes two or three)."""
import numpy as np
import pytest

import gpma_bfs_gb300 as G

pytestmark = pytest.mark.gpu


def test_path_of_40000_nodes(built_lib):
    n = 40_000
    u = np.arange(n - 1, dtype=np.uint64)
    g = G.GPMA(n)
    G.update_gpma(g, (u << np.uint64(32)) | (u + np.uint64(1)), np.ones(n - 1, np.uint8))
    levels, reached = G.gpma_bfs(g, n, 0, 0)
    assert reached == n and np.array_equal(levels, np.arange(1, n + 1))
    src = np.array([0, 100, n - 1], np.uint32)
    levels, reached = G.gpma_bfs_multi(g, src)
    for s, lv, r in zip(src.astype(np.int64), levels.astype(np.int64), reached):
        assert r == n - s and np.array_equal(lv, np.maximum(np.arange(n) - s + 1, 0))
    g.close()
