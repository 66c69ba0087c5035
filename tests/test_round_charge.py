"""What the served form charges its budget for a round's update buffers, against
what those buffers take."""
import numpy as np
import pytest

import gpma_bfs_gb300 as G

PER_KEY = 76  # window lists, batch and insertion buffers 71, buckets 1, look-back words 4


@pytest.mark.parametrize("lanes", [1, 2, 4])
def test_charge_per_key_and_lane(built_lib, lanes):
    def fixed(keys):
        s = G.Server(plan_only=True, hbm_budget_bytes=1 << 40, max_round_keys=keys, lanes=lanes)
        b = s.committed_bytes()
        s.close()
        return b

    assert fixed(1 << 20) == PER_KEY * lanes << 20
    assert fixed((1 << 20) + 1) - fixed(1 << 20) == PER_KEY * lanes


@pytest.mark.gpu
@pytest.mark.parametrize("sort", [0, 1])
def test_buffers_stay_within_the_charge(built_lib, sort):
    import torch

    n, rows = 1 << 22, 1 << 16
    rng = np.random.default_rng(8)
    k = (rng.integers(0, rows, n, dtype=np.uint64) << np.uint64(32)) | rng.integers(0, rows, n, dtype=np.uint64)
    keys = torch.from_numpy(k.view(np.int64)).cuda()
    values = torch.zeros(n, dtype=torch.uint8, device="cuda")  # deletes of nothing: the graph does not grow
    g = G.GPMA(rows)
    b = G.Batch()
    tuning = G.get_tuning()
    try:
        G.set_tuning(update_sort=sort)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        b.update_packed([g], keys, values, [0, n])
        torch.cuda.synchronize()
        taken = before - torch.cuda.mem_get_info()[0]
    finally:
        G.set_tuning(**tuning)
    # small tables and the allocator's 2 MB pages come on top
    assert 71 * n <= taken <= PER_KEY * n + (24 << 20)
    b.close()
    g.close()
