"""PageRank with a tolerance: it starts by adding per edge and goes over to gathering
where many more iterations are to come. Iterations and ranks are those of 64-bit
power iteration wherever the tolerance is met, and a tolerance met at once costs no
more than the iterations it took."""
import time

import numpy as np
import pytest

import gpma_bfs_gb300 as G

pytestmark = pytest.mark.gpu


def _graph(n, s, d):
    k = np.unique((s.astype(np.uint64) << np.uint64(32)) | d.astype(np.uint64))
    g = G.GPMA(n)
    G.update_gpma(g, np.random.default_rng(n).permutation(k), np.ones(len(k), np.uint8))
    return g, (k >> np.uint64(32)).astype(np.int64), (k & np.uint64(0xFFFFFFFF)).astype(np.int64)


def _power(n, s, d, damping, iterations):
    """(ranks after 0 .. iterations, change of each iteration)"""
    deg = np.bincount(s, minlength=n).astype(np.float64)
    r, ranks, change = np.full(n, 1.0 / n), [], []
    ranks.append(r)
    for _ in range(iterations):
        acc = np.bincount(d, weights=(np.where(deg > 0, r / np.maximum(deg, 1), 0.0))[s], minlength=n)
        nr = (1 - damping) / n + damping * (acc + r[deg == 0].sum() / n)
        change.append(np.abs(nr - r).sum())
        r = nr
        ranks.append(r)
    return ranks, change


@pytest.mark.parametrize("met", [1, 2, 3, 4, 5, 6, 9, 20])
@pytest.mark.parametrize("kind", ["rmat", "sparse", "hub", "tiny"])
def test_iterations_and_ranks(built_lib, kind, met):
    rng = np.random.default_rng(3)
    if kind == "rmat":
        n = 1 << 12
        s, d = G.gen_rmat(12, 8, seed=4)
    elif kind == "sparse":
        n = 30_000
        s, d = rng.integers(0, n, (2, 2 * n))
    elif kind == "hub":  # rows of several chunks
        n = 20_000
        s = np.r_[np.arange(n), rng.integers(0, n, n)]
        d = np.r_[np.full(n, 7), rng.integers(0, n, n)]
    else:  # arrays too small for the gathering
        n = 100
        s, d = rng.integers(0, n, (2, 300))
    g, s, d = _graph(n, np.asarray(s), np.asarray(d))
    ranks, change = _power(n, s, d, 0.85, met + 1)
    # between the changes of two iterations, so that rounding cannot move the end
    tol = float(np.sqrt(change[met - 1] * (change[met - 2] if met > 1 else 4 * change[0])))
    if tol < 1e-6:
        pytest.skip("the ranks' 32-bit rounding (2^-24 of their sum, 1, in every iteration) is a change of that size")
    for limit in (met, met + 3, 1000):
        got, its = G.pagerank(g, 0.85, limit, tol=tol)
        assert its == met
        np.testing.assert_allclose(got, ranks[met], rtol=2e-4, atol=1e-9)
    if met > 1:  # the limit first
        got, its = G.pagerank(g, 0.85, met - 1, tol=tol)
        assert its == met - 1
        np.testing.assert_allclose(got, ranks[met - 1], rtol=2e-4, atol=1e-9)
    g.close()


def test_a_tolerance_met_at_once_is_cheap(built_lib):
    """8 random cycles through all nodes: the uniform ranks are the fixed point."""
    import torch

    n = 1 << 18
    rng = np.random.default_rng(5)
    p = [rng.permutation(n) for _ in range(8)]
    g, _, _ = _graph(n, np.concatenate(p), np.concatenate([np.roll(x, 1) for x in p]))
    out = torch.zeros(n, dtype=torch.float32, device="cuda")

    def best(**kw):
        ts = []
        for _ in range(40):
            t = time.perf_counter()
            its = G.pagerank(g, 0.85, out=out, **kw)[1]
            ts.append(time.perf_counter() - t)
            assert its == 1
        return min(ts)

    # repeated edges are few, so the change is small, far below the tolerance
    assert best(iterations=100, tol=0.1) < 1.25 * best(iterations=1)
    g.close()


@pytest.mark.parametrize("n", [1, 2, 3, 5, 9, 20, 40])
def test_smallest_arrays(built_lib, n):
    """Arrays of 4 to 128 slots, on both sides of the smallest that is gathered."""
    rng = np.random.default_rng(n)
    s, d = rng.integers(0, n, (2, 2 * n))
    g, s, d = _graph(n, s, d)
    ranks, _ = _power(n, s, d, 0.85, 12)
    for its in (1, 3, 4, 12):
        got, done = G.pagerank(g, 0.85, its)
        assert done == its
        np.testing.assert_allclose(got, ranks[its], rtol=2e-4, atol=1e-9)
    g.close()
