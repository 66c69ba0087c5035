"""Digit passes of the batch sort with small and large tiles, at the batch size
where large tiles begin, against the oracle: one key less, exactly, one more and
a part tile more; one graph and several; keys over many and over few digits;
new keys repeated with differing values, whose order the sort keeps."""
import numpy as np
import pytest

from oracle.oracle import OracleGPMA

pytestmark = pytest.mark.gpu

TILE = 18 * 256  # keys of a large tile


@pytest.fixture
def one_cta_per_sm(built_lib):
    import torch

    import gpma_bfs_gb300 as G
    before = G.get_tuning()
    G.set_tuning(update_sort=1, update_blocks_per_sm=1)
    yield G, TILE * torch.cuda.get_device_properties(0).multi_processor_count
    G.set_tuning(**{f: before[f] for f in ("update_sort", "update_blocks_per_sm")})


def _keys(rng, rows, n):
    return (rng.integers(0, rows, n).astype(np.uint64) << np.uint64(32)) | rng.integers(0, rows, n).astype(np.uint64)


def _same(g, orc, ctx):
    assert g.geometry() == orc.geometry(), ctx
    for name, a, b in zip(("keys", "values", "row_offset"), g.export_layout(), orc.export_layout()):
        assert np.array_equal(a, b), f"{ctx}: {name}"


@pytest.mark.parametrize("rows", [700, 70000])
@pytest.mark.parametrize("more", [-1, 0, 1, TILE - 1, TILE + 31])
def test_one_graph(one_cta_per_sm, rows, more):
    G, limit = one_cta_per_sm
    rng = np.random.default_rng(rows + more)
    g, orc = G.GPMA(rows), OracleGPMA(rows, threads=4)
    n = limit + more
    k = _keys(rng, rows, n)
    v = rng.integers(0, 4, n).astype(np.uint8)
    G.update_gpma(g, k, v)
    orc.update(k, v)
    _same(g, orc, "load")
    # in place, each key once: repeats of a live key have no order
    k = rng.permutation(np.unique(np.concatenate([k, _keys(rng, rows, 1000)])))
    v = rng.integers(0, 3, len(k)).astype(np.uint8)
    G.update_gpma(g, k, v)
    orc.update(k, v)
    _same(g, orc, "update")
    g.close()


@pytest.mark.parametrize("parts", [(1, 1, 1), (0, 1, 5), (100, 1, 0.001)])
@pytest.mark.parametrize("more", [-1, 0, 77])
def test_many_graphs(one_cta_per_sm, parts, more):
    G, limit = one_cta_per_sm
    rng = np.random.default_rng(more + 1)
    n = limit + more
    sizes = [int(n * p / sum(parts)) for p in parts]
    sizes[1] += n - sum(sizes)
    rows = [3000, 20000, 900]
    gs, orcs = [G.GPMA(r) for r in rows], [OracleGPMA(r, threads=4) for r in rows]
    b = G.Batch()
    ks = [_keys(rng, r, m) for r, m in zip(rows, sizes)]
    vs = [rng.integers(0, 4, m).astype(np.uint8) for m in sizes]
    b.update(gs, ks, vs)
    for o, g, k, v in zip(orcs, gs, ks, vs):
        if len(k):
            o.update(k, v)
        _same(g, o, f"{len(k)} keys")
    b.close()
    for g in gs:
        g.close()


@pytest.mark.parametrize("more", [-1, 0])
def test_large_batches_of_one_graph(built_lib, more):
    """The batch size where digit passes replace the buckets."""
    import gpma_bfs_gb300 as G
    rng = np.random.default_rng(9)
    rows, n = 300000, (1 << 22) + more
    g, orc = G.GPMA(rows), OracleGPMA(rows, threads=8)
    k = np.unique(_keys(rng, rows, 5_000_000))
    for step, (keys, value) in enumerate(((k, 1), (rng.permutation(k)[:n], 2), (rng.permutation(k)[:n], 0),
                                          (rng.permutation(np.unique(_keys(rng, rows, n + 9000)))[:n], 3))):
        v = np.full(len(keys), value, np.uint8)
        G.update_gpma(g, keys, v)
        orc.update(keys, v)
        _same(g, orc, f"step {step}")
    g.close()
