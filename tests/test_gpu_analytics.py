"""PageRank and weakly connected components over the gapped array, against
plain CPU computations on the graph's live edge set (taken from the oracle
after the same updates, tombstones included)."""
import numpy as np
import pytest

from oracle.oracle import OracleGPMA

pytestmark = pytest.mark.gpu


def _graph():
    import gpma_bfs_gb300 as G

    n = 1 << 12
    src, dst = G.gen_rmat(12, 6, seed=21)
    keys = G.edges_to_keys(src, dst)
    g, o = G.GPMA(n), OracleGPMA(n, threads=2)
    for k, v in ((keys, np.ones(len(keys), np.uint8)), (keys[::3], np.zeros(len(keys[::3]), np.uint8))):
        G.update_gpma(g, k, v)
        o.update(k, v)
    live = o.compact_keys()
    s, d = (live >> np.uint64(32)).astype(np.int64), (live & np.uint64(0xFFFFFFFF)).astype(np.int64)
    edge = (d != 0xFFFFFFFF) & (s < n) & (d < n)
    return G, g, n, s[edge], d[edge]


def test_components_equal_scipy(built_lib):
    sp = pytest.importorskip("scipy.sparse")
    csgraph = pytest.importorskip("scipy.sparse.csgraph")
    G, g, n, s, d = _graph()
    labels, count, rounds = G.components(g)
    a = sp.csr_matrix((np.ones(len(s)), (s, d)), shape=(n, n))
    ncomp, lab = csgraph.connected_components(a, directed=True, connection="weak")
    # canonical labels: the smallest node id of each component
    first = np.full(ncomp, n, np.int64)
    np.minimum.at(first, lab, np.arange(n))
    assert count == ncomp and rounds >= 1
    assert np.array_equal(labels, first[lab].astype(np.uint32))
    g.close()


def _pagerank_f64(n, s, d, damping, iterations):
    deg = np.bincount(s, minlength=n).astype(np.float64)
    r = np.full(n, 1.0 / n)
    for _ in range(iterations):
        contrib = np.where(deg > 0, r / np.maximum(deg, 1), 0.0)
        dangling = r[deg == 0].sum()
        acc = np.bincount(d, weights=contrib[s], minlength=n)
        r = (1 - damping) / n + damping * (acc + dangling / n)
    return r


def test_pagerank_matches_float64_power_iteration(built_lib):
    G, g, n, s, d = _graph()
    want = _pagerank_f64(n, s, d, 0.85, 30)
    got, iters = G.pagerank(g, 0.85, 30)
    assert iters == 30
    # float32 ranks with float atomics: within 2e-4 relative (+1e-8 absolute) of float64
    np.testing.assert_allclose(got, want, rtol=2e-4, atol=1e-8)
    assert abs(got.sum() - 1.0) < 1e-3
    # with a tolerance the iteration stops early and is still close to the fixed point
    conv, it2 = G.pagerank(g, 0.85, 500, tol=1e-7)
    assert it2 < 500
    np.testing.assert_allclose(conv, _pagerank_f64(n, s, d, 0.85, 200), rtol=1e-3, atol=1e-8)
    g.close()


def test_analytics_on_device_outputs_and_empty_edges(built_lib):
    import torch

    import gpma_bfs_gb300 as G

    g = G.GPMA(100)  # guards only: every node is isolated and dangling
    lab = torch.zeros(100, dtype=torch.int32, device="cuda")
    _, count, _ = G.components(g, lab)
    assert count == 100 and np.array_equal(lab.cpu().numpy(), np.arange(100))
    r = torch.zeros(100, dtype=torch.float32, device="cuda")
    G.pagerank(g, 0.85, 5, out=r)
    np.testing.assert_allclose(r.cpu().numpy(), np.full(100, 0.01), rtol=1e-5)
    g.close()


def _labels(n, s, d):
    """Smallest node id of each node's component, by label propagation with pointer jumping."""
    lab = np.arange(n)
    while True:
        new = lab.copy()
        np.minimum.at(new, s, lab[d])
        np.minimum.at(new, d, lab[s])
        new = new[new]
        if np.array_equal(new, lab):
            return lab
        lab = new


@pytest.mark.parametrize("shape", ["one", "pair", "path_up", "path_down", "star", "late_edges", "sparse"])
def test_components_link_shapes(built_lib, shape):
    """Tree shapes at the edges of the linking: arrays of 4 slots, long chains in
    both id orders, one hub, rows whose only joining edges lie behind the sampled
    slots, many small components; deleted edges link nothing."""
    import gpma_bfs_gb300 as G

    rng = np.random.default_rng(5)
    n = {"one": 1, "pair": 2, "star": 3001, "sparse": 5000}.get(shape, 4097)
    i = np.arange(n - 1)
    s, d = {
        "one": (i, i),
        "pair": (np.array([1]), np.array([0])),
        "path_up": (i, i + 1),
        "path_down": (i + 1, i),
        "star": (np.full(n - 1, n - 1), i),
        "late_edges": (i // 40 * 40, i + 1),
        "sparse": (rng.integers(0, n, n // 3), rng.integers(0, n, n // 3)),
    }[shape]
    g = G.GPMA(n)
    if len(s):
        keys = np.unique(G.edges_to_keys(s.astype(np.uint32), d.astype(np.uint32)))
        gone = rng.random(len(keys)) < (0.02 if n > 2 else 0)
        G.update_gpma(g, keys, np.ones(len(keys), np.uint8))
        G.update_gpma(g, keys[gone], np.zeros(int(gone.sum()), np.uint8))
        keys = keys[~gone]
        s, d = (keys >> np.uint64(32)).astype(np.int64), (keys & np.uint64(0xFFFFFFFF)).astype(np.int64)
    want = _labels(n, s, d)
    got, count, _ = G.components(g)
    assert np.array_equal(got, want) and count == len(np.unique(want))
    g.close()


@pytest.mark.parametrize("iterations,tol", [(3, 0.0), (4, 0.0), (25, 0.0), (400, 1e-4)])
def test_pagerank_row_lengths(built_lib, iterations, tol):
    """In-edge rows at the edges of the gathered layout (none, one step, the
    longest short row, one chunk, one more than a chunk, several chunks), on both sides of the iteration count that lays the in-edges out.
    float32 sums of up to 9,000 positive terms in partial sums, 25 iterations:
    well under the 2e-4 of the test above."""
    import gpma_bfs_gb300 as G

    n = 12000
    lens = {0: 0, 1: 1, 2: 15, 3: 16, 4: 17, 5: 63, 6: 64, 7: 65, 8: 4095, 9: 4096, 10: 4097, 11: 9000, n - 1: 300}
    rng = np.random.default_rng(3)
    s = np.concatenate([rng.choice(np.arange(20, n - 20), k, replace=False) for k in lens.values()])
    d = np.concatenate([np.full(k, v) for v, k in lens.items()])
    keys = G.edges_to_keys(s.astype(np.uint32), d.astype(np.uint32))
    gone = np.sort(rng.choice(len(keys), 50, replace=False))
    g = G.GPMA(n)
    G.update_gpma(g, np.concatenate([keys, G.edges_to_keys(np.uint32([30]), np.uint32([31]))]),
                  np.ones(len(keys) + 1, np.uint8))
    G.update_gpma(g, keys[gone], np.zeros(50, np.uint8))
    # lengths stay exact: the deleted edges come back, one other edge goes
    G.update_gpma(g, np.concatenate([keys[gone], G.edges_to_keys(np.uint32([30]), np.uint32([31]))]),
                  np.concatenate([np.ones(50, np.uint8), np.zeros(1, np.uint8)]))
    got, its = G.pagerank(g, 0.85, iterations, tol=tol)
    if tol:  # the first iteration whose change is below tol, give or take the rounding of the sum
        r = [_pagerank_f64(n, s, d, 0.85, t) for t in range(80)]
        change = [np.abs(b - a).sum() for a, b in zip(r, r[1:])]
        assert change[its - 1] < 2 * tol and (its < 2 or change[its - 2] > tol / 2)
    else:
        assert its == iterations
    np.testing.assert_allclose(got, _pagerank_f64(n, s, d, 0.85, its), rtol=2e-4, atol=1e-9)
    again, _ = G.pagerank(g, 0.85, iterations, tol=tol)
    np.testing.assert_allclose(again, got, rtol=2e-4)
    g.close()
