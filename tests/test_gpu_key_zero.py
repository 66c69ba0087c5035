"""Edge 0 -> 0, whose key 0 is also the key of the bulk rebuild's gaps: inserted
into, deleted from and modified in arrays with such gaps in their first leaf, by
every path a batch can take, the array stays a sorted list of exactly the edges
of a plain set, and the next bulk rebuild keeps it so."""
import numpy as np
import pytest

import gpma_bfs_gb300 as G

pytestmark = pytest.mark.gpu

BULK = 5_000_000  # insertions of a bulk rebuild, rows of a graph created with its gaps
NONE32 = 0xFFFFFFFF


def _check(g, edges, ctx):
    """edges: the live edges' keys in order, and their values."""
    keys, vals, ro = g.export_layout()
    live = (vals != 0) & (keys != np.uint64(0xFFFFFFFFFFFFFFFF))
    k, v = keys[live], vals[live]
    real = k < np.uint64(0xFFFFFFFFFFFFFFFE)  # without the initial entries
    assert np.all(k[real][1:] > k[real][:-1]), f"{ctx}: not sorted"
    edge = real & ((k & np.uint64(NONE32)) != np.uint64(NONE32))
    assert np.array_equal(k[edge], edges[0]), f"{ctx}: edges"
    assert np.array_equal(v[edge], edges[1]), f"{ctx}: values"
    guards = (np.arange(g.row_num, dtype=np.uint64) << np.uint64(32)) | np.uint64(NONE32)
    assert np.array_equal(keys[ro[1:]], guards) and ro[0] == 0, f"{ctx}: rows"
    assert g.validate() == 0, ctx


def _apply(edges, k, v):
    o = np.argsort(k)
    k, v = k[o], v[o]
    old, val = edges
    at = np.searchsorted(old, k)
    if len(old):
        hit = at < len(old)
        hit[hit] = old[at[hit]] == k[hit]
        keep = np.ones(len(old), bool)
        keep[at[hit]] = False
        old, val = old[keep], val[keep]
    k, v = k[v != 0], v[v != 0]
    at = np.searchsorted(old, k)
    return np.insert(old, at, k), np.insert(val, at, v)


def _spread(rng, rows, n):
    """n distinct keys without 0."""
    k = np.unique((rng.integers(0, rows, n + n // 8, dtype=np.uint64) << np.uint64(32)) |
                  rng.integers(1, 1 << 22, n + n // 8, dtype=np.uint64))
    return rng.permutation(k)[:n]


def _update(g, k, v, how):
    if how == "batch":
        other = G.GPMA(50)
        b = G.Batch()
        b.update([other, g], [np.array([5], np.uint64), k], [np.ones(1, np.uint8), v])
        b.close()
        other.close()
    else:
        G.update_gpma(g, k, v)


@pytest.mark.parametrize("gaps, n, how", [("created", 1, "small"), ("created", 4096, "small"),
                                          ("created", 4097, "general"), ("created", 60_000, "digits"),
                                          ("created", 60_000, "batch"), ("created", BULK + 10, "bulk"),
                                          ("loaded", 1, "small"), ("loaded", 5000, "general")])
def test_edge_zero_among_gaps(built_lib, gaps, n, how):
    rng = np.random.default_rng(n)
    rows = BULK if gaps == "created" else 3000
    g = G.GPMA(rows)
    edges = (np.zeros(0, np.uint64), np.zeros(0, np.uint8))
    if gaps == "loaded":
        k = _spread(rng, rows, BULK + 1)
        G.update_gpma(g, k, np.ones(len(k), np.uint8))
        edges = _apply(edges, k, np.ones(len(k), np.uint8))
    first = g.export_layout()
    leaf = g.segment_length
    assert np.any(first[0][1:leaf] == 0), "no gap with key 0 in the first leaf"
    tuning = G.get_tuning()
    try:
        if how == "digits":
            G.set_tuning(update_sort=1)
        zero = np.zeros(1, np.uint64)
        # a delete of the edge that is not there changes nothing
        _update(g, zero, np.zeros(1, np.uint8), how)
        assert all(np.array_equal(a, b) for a, b in zip(first, g.export_layout()))
        # insert, modify, delete and revive it, in batches of n keys
        for step, value in enumerate((2, 3, 0, 1)):
            k = np.concatenate([zero, _spread(rng, rows, n - 1)])
            v = np.full(len(k), 1, np.uint8)
            v[0] = value
            o = rng.permutation(len(k))
            _update(g, k[o], v[o], how)
            edges = _apply(edges, k, v)
            _check(g, edges, f"{how}, step {step}")
            if how == "bulk" and step == 1:
                break
    finally:
        G.set_tuning(**tuning)
    if n in (1, 4097):
        k = _spread(rng, rows, BULK + 5)
        G.update_gpma(g, k, np.ones(len(k), np.uint8))
        edges = _apply(edges, k, np.ones(len(k), np.uint8))
        _check(g, edges, f"{how}, next bulk rebuild")
    lv, _ = G.gpma_bfs(g, rows, 0, 0)
    first_row = edges[0][edges[0] < np.uint64(1 << 32)]
    first_row = first_row[(first_row > 0) & (first_row < rows)].astype(np.int64)
    want = np.zeros(rows, bool)
    want[first_row] = True
    assert lv[0] == 1 and np.array_equal(lv == 2, want), "levels"
    g.close()
