"""A search that fails on the device leaves host arrays as they were; the next one
writes every level, whatever the failed one left in a device array."""
import numpy as np
import pytest

import gpma_bfs_gb300 as G

pytestmark = pytest.mark.gpu


def test_levels_of_a_stalled_search(built_lib):
    import torch

    n = 3000
    rng = np.random.default_rng(2)
    k = np.unique((rng.integers(0, n, 9000).astype(np.uint64) << np.uint64(32)) | rng.integers(0, n, 9000).astype(np.uint64))
    g = G.GPMA(n)
    G.update_gpma(g, k, np.ones(len(k), np.uint8))
    want, reached = G.gpma_bfs(g, n, 0, 5)
    host = np.full(n, 7, np.uint32)
    pinned = torch.full((n,), 7, dtype=torch.int32).pin_memory()
    device = torch.full((n,), 7, dtype=torch.int32, device="cuda")
    try:
        G.set_test_hooks(bfs_stall=1, wait_limit_us=20_000)
        for levels in (host, pinned, device):
            with pytest.raises(G.GPMAError) as e:
                G.gpma_bfs(g, n, 0, 5, levels)
            assert e.value.status == 5  # GPMA_ERR_TIMEOUT
    finally:
        G.set_test_hooks(bfs_stall=0, wait_limit_us=0)
    assert np.all(host == 7) and bool((pinned == 7).all())
    for levels in (host, pinned, device):
        assert G.gpma_bfs(g, n, 0, 5, levels)[1] == reached
        got = levels if isinstance(levels, np.ndarray) else levels.cpu().numpy()
        assert np.array_equal(got, want)
    g.close()
