"""Multi-source BFS against the oracle's single searches: graphs of a few nodes
that share a warp's 32 nodes, rows at the edges of the walk's steps and chunks,
1 to 64 sources, levels on the host, on the device and left out, on both sides
of the switch to the whole-array sweep."""
import numpy as np
import pytest

from oracle.oracle import OracleGPMA

pytestmark = pytest.mark.gpu


def _graphs(G, rng):
    """(gpu graph, oracle, nodes): tiny ones between larger ones."""
    out = []
    for n, m in ((1, 0), (2, 1), (5, 6), (31, 60), (3, 2), (700, 2500), (33, 200), (1, 0), (1500, 9000)):
        src, dst = rng.integers(0, n, m), rng.integers(0, n, m)
        if n >= 700:  # rows of 63 .. 66 and 127 .. 130 and 400 edges
            hubs = [np.full(k, i * 7) for i, k in enumerate((63, 64, 65, 66, 127, 128, 129, 130, 400))]
            src = np.concatenate([src, *hubs])
            dst = np.concatenate([dst, *[rng.choice(n, len(h), replace=False) for h in hubs]])
        keys = np.unique(G.edges_to_keys(src.astype(np.uint32), dst.astype(np.uint32)))
        g, o = G.GPMA(n), OracleGPMA(n, threads=2)
        if len(keys):
            gone = keys[rng.random(len(keys)) < 0.05]
            for k, v in ((keys, 1), (gone, 0)):
                if len(k):
                    vals = np.full(len(k), v, np.uint8)
                    G.update_gpma(g, k, vals)
                    o.update(k, vals)
        out.append((g, o, n))
    return out


@pytest.mark.parametrize("dense_div", [0, 8, 1 << 20])
@pytest.mark.parametrize("k", [1, 31, 33, 64])
def test_levels_and_counts_equal_oracle(built_lib, k, dense_div):
    import torch

    import gpma_bfs_gb300 as G

    rng = np.random.default_rng(100 + k)
    gs = _graphs(G, rng)
    sources = [rng.integers(0, n, k).astype(np.uint32) for _, _, n in gs]
    want = [[o.bfs(int(s)) for s in src] for (_, o, _), src in zip(gs, sources)]
    old = G.set_tuning(ms_dense_div=dense_div)
    try:
        b = G.Batch()
        levels, reached = b.bfs_multi([g for g, _, _ in gs], sources, levels=True)
        counts = b.bfs_multi([g for g, _, _ in gs], sources)[1]
        for i, w in enumerate(want):
            assert np.array_equal(levels[i], np.stack([x[0] for x in w])), f"graph {i}"
            assert [int(x) for x in reached[i]] == [x[1] for x in w] == [int(x) for x in counts[i]]
        for i in (3, 5, 8):
            g, _, n = gs[i]
            out = torch.full((k, n), -1, dtype=torch.int32, device="cuda")  # every entry is written
            _, r = G.gpma_bfs_multi(g, sources[i], out)
            assert np.array_equal(out.cpu().numpy().astype(np.uint32), np.stack([x[0] for x in want[i]]))
            assert [int(x) for x in r] == [x[1] for x in want[i]]
        b.close()
    finally:
        G.set_tuning(**old)
    for g, _, _ in gs:
        g.close()


@pytest.mark.parametrize("k", [5, 40])
@pytest.mark.parametrize("n", [62, 63, 64, 65, 300])
def test_levels_of_long_paths(built_lib, k, n):
    """Depths around the number of levels the bit planes hold (63) and far past it."""
    import gpma_bfs_gb300 as G

    i = np.arange(n - 1, dtype=np.uint32)
    keys = np.concatenate([G.edges_to_keys(i, i + 1), G.edges_to_keys(np.uint32([n - 1]), np.uint32([0]))])
    g = G.GPMA(n)
    G.update_gpma(g, keys, np.ones(len(keys), np.uint8))
    src = (np.arange(k) * 7 % n).astype(np.uint32)
    levels, reached = G.gpma_bfs_multi(g, src)
    want = (np.arange(n)[None, :] - src[:, None].astype(np.int64)) % n + 1
    assert np.array_equal(levels, want) and all(int(r) == n for r in reached)
    g.close()
