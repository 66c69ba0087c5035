"""Small batches of one graph (ordered, located and grouped with one grid
barrier) against the oracle, on both sides of the size where the general phases
take over: sizes around a warp, a CTA, the grid's warps and the limit; batches
spread over the array, in one row (windows that climb the tree), around the
array's ends; inserts, repeats, modifies, deletes of live, dead and absent keys,
revivals; arrays from 4 slots up; device, pinned and pageable batches."""
import numpy as np
import pytest

from oracle.oracle import OracleGPMA
from replay import GpuAdapter

pytestmark = pytest.mark.gpu

LIMIT = 4096


def _same(gpu, orc, ctx):
    assert gpu.geometry() == orc.geometry(), ctx
    for name, a, b in zip(("keys", "values", "row_offset"), gpu.export_layout(), orc.export_layout()):
        assert np.array_equal(a, b), f"{ctx}: {name}"
    assert gpu.g.validate() == 0, ctx


def _both(gpu, orc, k, v, ctx):
    gpu.update(k, v)
    orc.update(k, v)
    _same(gpu, orc, ctx)


def _keys(rng, shape, rows, n):
    if shape == "spread":
        s, d = rng.integers(0, rows, n), rng.integers(0, rows, n)
    elif shape == "one_row":
        s, d = np.full(n, rows // 3), rng.permutation(5 * n)[:n]
    else:  # ends
        s = np.where(rng.random(n) < 0.5, 0, rows - 1)
        d = rng.integers(0, 4 * n, n)
    return (s.astype(np.uint64) << np.uint64(32)) | d.astype(np.uint64)


@pytest.mark.parametrize("shape", ["spread", "one_row", "ends"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 255, 257, 2431, 2433, LIMIT - 1, LIMIT, LIMIT + 1])
def test_small_batches_equal_oracle(built_lib, shape, n):
    rng = np.random.default_rng(n)
    rows = 3000
    gpu, orc = GpuAdapter(rows), OracleGPMA(rows, threads=4)
    load = np.unique(_keys(rng, "spread", rows, 30000))
    _both(gpu, orc, rng.permutation(load), np.ones(len(load), np.uint8), "load")
    fresh = _keys(rng, shape, rows, n)
    old = rng.choice(load, n)
    for step, (k, v) in enumerate((
            (fresh, 1),
            (np.concatenate([fresh[: n // 2], old[: n - n // 2]]), 0),  # delete live keys, some twice
            (rng.permutation(np.concatenate([fresh[: n // 3], old[: n - n // 3]])), 2),  # revive and modify
            (_keys(rng, shape, rows, n), 0))):  # mostly absent
        _both(gpu, orc, k, np.full(len(k), v, np.uint8), f"step {step}")
    mixed = np.unique(np.concatenate([_keys(rng, shape, rows, n // 2 + 1), old[: n // 2]]))[:n]
    _both(gpu, orc, rng.permutation(mixed), rng.integers(0, 3, len(mixed)).astype(np.uint8), "mixed")
    repeats = np.repeat(_keys(rng, shape, rows, n // 2 + 1), 2)[:n]
    _both(gpu, orc, repeats, np.ones(n, np.uint8), "repeats")
    gpu.close()


@pytest.mark.parametrize("rows", [1, 2, 3, 5])
def test_small_batches_grow_tiny_arrays(built_lib, rows):
    rng = np.random.default_rng(rows)
    gpu, orc = GpuAdapter(rows), OracleGPMA(rows, threads=1)
    for step, n in enumerate((1, 1, 2, 3, 40, 300)):
        k = _keys(rng, "spread", rows, n) * np.uint64(1) + np.arange(n, dtype=np.uint64)
        _both(gpu, orc, k, np.ones(n, np.uint8), f"step {step}")
    gpu.close()


def test_small_batches_from_device_pinned_and_rejected(built_lib):
    import torch

    import gpma_bfs_gb300 as G

    rng = np.random.default_rng(8)
    rows = 500
    gpu, orc = GpuAdapter(rows), OracleGPMA(rows, threads=2)
    for where in ("device", "pinned", "pageable"):
        k = np.unique(_keys(rng, "spread", rows, 700))
        v = np.ones(len(k), np.uint8)
        tk, tv = torch.from_numpy(k.view(np.int64)), torch.from_numpy(v)
        if where == "device":
            tk, tv = tk.cuda(), tv.cuda()
        elif where == "pinned":
            tk, tv = tk.pin_memory(), tv.pin_memory()
        G.update_gpma(gpu.g, tk, tv)
        orc.update(k, v)
        _same(gpu, orc, where)
        bad = np.append(k[:5], np.uint64((3 << 32) | 0xFFFFFFFF))
        with pytest.raises(G.GPMAError):
            G.update_gpma(gpu.g, bad, np.ones(6, np.uint8))
        _same(gpu, orc, where + " after a rejected batch")
    gpu.close()
