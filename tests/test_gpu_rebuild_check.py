"""A bulk rebuild over an array that is not sorted (its halves swapped behind the
library's back) is reported as GPMA_ERR_DEVICE naming the split check, in the
product build too; the library goes on working."""
import numpy as np
import pytest

import gpma_bfs_gb300 as G

pytestmark = pytest.mark.gpu

BULK = 5_000_000
ROWS = 3000


def _keys(seed):
    rng = np.random.default_rng(seed)
    k = np.unique((rng.integers(0, ROWS, BULK + BULK // 8, dtype=np.uint64) << np.uint64(32)) |
                  rng.integers(1, 1 << 22, BULK + BULK // 8, dtype=np.uint64))
    return rng.permutation(k)[:BULK + 3]


def _view(ptr, n, typestr):
    import torch

    class View:
        __cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 3}

    return torch.as_tensor(View(), device="cuda")


def test_unsorted_array_is_reported(built_lib):
    import torch

    ones = np.ones(BULK + 3, np.uint8)
    first, second = _keys(1), _keys(2)
    g = G.GPMA(ROWS)
    G.update_gpma(g, first, ones)
    size = g.get_size()
    kp, vp, _ = g.device_arrays()
    for a in (_view(kp, size, "<i8"), _view(vp, size, "|u1")):
        a.copy_(torch.roll(a, size // 2))
    torch.cuda.synchronize()
    with pytest.raises(G.GPMAError) as e:
        G.update_gpma(g, second, ones)
    assert e.value.status == 7 and "site 5" in str(e.value), str(e.value)
    g.close()
    h = G.GPMA(ROWS)
    G.update_gpma(h, first, ones)
    G.update_gpma(h, second, ones)
    keys, vals, _ = h.export_layout()
    edge = (vals != 0) & ((keys & np.uint64(0xFFFFFFFF)) < np.uint64(1 << 22))
    assert np.array_equal(keys[edge], np.union1d(first, second))
    h.close()
