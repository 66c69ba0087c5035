"""Updates of several graphs in one launch whose levels have more or fewer windows
than are dispatched by ranges (160 per CTA): graphs of different segment lengths,
every layout against the oracle."""
import numpy as np
import pytest

import gpma_bfs_gb300 as G
from oracle.oracle import OracleGPMA

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [0, 1])  # 304 and 152 CTAs
@pytest.mark.parametrize("keys", [3_000, 60_000, 240_000])
def test_levels_of_many_graphs(built_lib, blocks, keys):
    rng = np.random.default_rng(keys + blocks)
    rows = [40, 700, 9_000, 90_000, 5, 200_000]
    share = [0.02, 0.08, 0.2, 0.3, 0.001, 0.4]
    tuning = G.get_tuning()
    b = G.Batch()
    gpu = [G.GPMA(r) for r in rows]
    orc = [OracleGPMA(r, threads=4) for r in rows]
    try:
        G.set_tuning(update_blocks_per_sm=blocks)
        for step in range(4):
            ks, vs = [], []
            for r, f in zip(rows, share):
                n = max(1, int(f * keys))
                k = np.unique((rng.integers(0, r, n, dtype=np.uint64) << np.uint64(32)) |
                              rng.integers(0, max(r, 4 * n), n, dtype=np.uint64))
                k = rng.permutation(k)
                ks.append(k)
                vs.append(rng.integers(0, 3, len(k)).astype(np.uint8) if step else np.ones(len(k), np.uint8))
            b.update(gpu, ks, vs)
            for i, (g, o) in enumerate(zip(gpu, orc)):
                o.update(ks[i], vs[i])
                ctx = f"step {step}, graph {i}"
                assert g.geometry() == o.geometry(), ctx
                for x, y in zip(g.export_layout(), o.export_layout()):
                    assert np.array_equal(x, y), ctx
                assert g.validate() == 0, ctx
    finally:
        G.set_tuning(**tuning)
        b.close()
        for g in gpu:
            g.close()
