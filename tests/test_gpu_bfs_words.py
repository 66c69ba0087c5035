"""Single-source BFS against the oracle at the edges of its walk: rows at the
limits of a short row, a step and a chunk, node counts around a bitmap word,
one CTA and many, hubs whose chunks overflow a CTA's list, the whole-array
sweep, and levels on the host, on the device and at an odd 4-byte offset."""
import numpy as np
import pytest

from oracle.oracle import OracleGPMA

pytestmark = pytest.mark.gpu


def _pair(n, src, dst):
    import gpma_bfs_gb300 as G

    keys = np.unique(G.edges_to_keys(src.astype(np.uint32), dst.astype(np.uint32)))
    g, o = G.GPMA(n), OracleGPMA(n, threads=4)
    gone = keys[::17]
    for k, v in ((keys, 1), (gone, 0)):
        if len(k):
            vals = np.full(len(k), v, np.uint8)
            G.update_gpma(g, k, vals)
            o.update(k, vals)
    return G, g, o


def _check(G, g, o, n, sources):
    import torch

    for s in sources:
        want, reached = o.bfs(int(s))
        got, r = G.gpma_bfs(g, n, 0, int(s))
        assert r == reached and np.array_equal(got, want)
        dev = torch.full((n + 1,), -1, dtype=torch.int32, device="cuda")
        for out in (dev[:n], dev[1:]):
            _, r = G.gpma_bfs(g, n, 0, int(s), out)
            assert r == reached and np.array_equal(out.cpu().numpy().view(np.uint32), want)


@pytest.mark.parametrize("dense_div", [0, 2, 1 << 20])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 700, 5000])
def test_bfs_rows_and_words(built_lib, n, dense_div):
    rng = np.random.default_rng(n)
    m = 4 * n
    src, dst = rng.integers(0, n, m), rng.integers(0, n, m)
    if n >= 700:
        lens = [l for l in (15, 31, 32, 47, 63, 64, 65, 127, 128, 129, 255, 256, 257, 600) if l <= n]
        src = np.concatenate([src, *[np.full(l, 3 * i) for i, l in enumerate(lens)]])
        dst = np.concatenate([dst, *[rng.choice(n, l, replace=False) for l in lens]])
    G, g, o = _pair(n, src, dst)
    old = G.set_tuning(bfs_dense_div=dense_div)
    try:
        _check(G, g, o, n, rng.integers(0, n, 4))
    finally:
        G.set_tuning(**old)
    g.close()


@pytest.mark.parametrize("blocks", [1, 8])
def test_bfs_hubs_overflow_a_ctas_chunk_list(built_lib, blocks):
    """Rows of 40,000 edges in neighbouring nodes: with one CTA per SM a warp's
    words hold more chunks than the CTA's list, so they take the grid's list."""
    n = 60000
    rng = np.random.default_rng(9)
    hubs = [0, 1, 2, 31, 32, 5000]
    src = np.concatenate([np.repeat(hubs, 40000), rng.integers(0, n, 30000)])
    dst = np.concatenate([np.concatenate([rng.choice(n, 40000, replace=False) for _ in hubs]), rng.integers(0, n, 30000)])
    G, g, o = _pair(n, src, dst)
    old = G.set_tuning(bfs_blocks_per_sm=blocks)
    try:
        _check(G, g, o, n, [0, 7, 31, 59999])
    finally:
        G.set_tuning(**old)
    g.close()


def test_step_leaves_levels_alone_when_its_batch_is_refused(built_lib):
    import torch

    n = 64
    G, g, o = _pair(n, np.arange(63), np.arange(1, 64))
    step = G.Step(g)
    out = torch.full((n,), -5, dtype=torch.int32, device="cuda")
    ok = np.array([3], np.uint64)
    step.run(ok, np.ones(1, np.uint8), 0, out)
    o.update(ok, np.ones(1, np.uint8))
    assert np.array_equal(out.cpu().numpy().view(np.uint32), o.bfs(0)[0])
    out.fill_(-5)
    with pytest.raises(G.GPMAError):
        step.run(np.array([0xFFFFFFFF], np.uint64), np.ones(1, np.uint8), 0, out)
    assert bool((out == -5).all())
    o.update(ok, np.zeros(1, np.uint8))
    assert step.run(ok, np.zeros(1, np.uint8), 0, out) == o.bfs(0)[1]
    step.close()
    g.close()
