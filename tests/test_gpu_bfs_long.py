"""Searches of more levels than the first kernel takes (64): the levels on both
sides of that line, long thin graphs whose levels end with one barrier, levels too
large for that in between, through every call that searches one graph."""
import ctypes
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import gpma_bfs_gb300 as G

pytestmark = pytest.mark.gpu


def _graph(n, src, dst):
    g = G.GPMA(n)
    k = np.unique((np.asarray(src).astype(np.uint64) << np.uint64(32)) | np.asarray(dst).astype(np.uint64))
    G.update_gpma(g, np.random.default_rng(n).permutation(k), np.ones(len(k), np.uint8))
    return g


def _check(g, n, source, want):
    levels, reached = G.gpma_bfs(g, n, 0, source)
    assert np.array_equal(levels, want) and reached == np.count_nonzero(want)


@pytest.mark.parametrize("n", [2, 62, 63, 64, 65, 66, 67, 129, 3000])
def test_paths_around_the_line(built_lib, n):
    g = _graph(n + 1, np.arange(n - 1), np.arange(1, n))  # node n stays alone
    for s in (0, 1, n - 1):
        want = np.where(np.arange(n + 1) >= s, np.arange(n + 1) - s + 1, 0)
        want[n] = 0
        _check(g, n + 1, s, want)
    g.close()


@pytest.mark.parametrize("m", [40, 100, 333])
def test_grids(built_lib, m):
    i = np.arange(m * m)
    a, b = i[i % m < m - 1], i[i < m * m - m]
    g = _graph(m * m, np.r_[a, a + 1, b, b + m], np.r_[a + 1, a, b + m, b])
    x, y = i % m, i // m
    for s in (0, m * m - 1, m * (m // 3) + 2):
        _check(g, m * m, s, np.abs(x - s % m) + np.abs(y - s // m) + 1)
    g.close()


def _hubs(h, leaves):
    """A chain of h hubs, each with its own leaves; a level per hub."""
    hub = np.arange(h)
    src = np.r_[hub[:-1], np.repeat(hub, leaves)]
    dst = np.r_[hub[1:], h + np.arange(h * leaves)]
    want = np.r_[hub + 1, np.repeat(hub + 2, leaves)]
    return h * (leaves + 1), src, dst, want


@pytest.mark.parametrize("h, leaves", [(70, 1), (100, 3000), (90, 40_000)])
def test_levels_with_long_rows(built_lib, h, leaves):
    n, src, dst, want = _hubs(h, leaves)
    g = _graph(n, src, dst)
    _check(g, n, 0, want)
    tuning = G.get_tuning()
    try:
        G.set_tuning(bfs_dense_div=4)
        _check(g, n, 0, want)
        G.set_tuning(bfs_dense_div=0, bfs_blocks_per_sm=1)
        _check(g, n, 0, want)
    finally:
        G.set_tuning(**tuning)
    g.close()


@pytest.mark.parametrize("cap", [0, 1, 37])
def test_without_allocation(built_lib, cap):
    import torch

    n, src, dst, want = _hubs(100, 3000)
    g = _graph(n, src, dst)
    levels = torch.full((n,), 9, dtype=torch.int32, device="cuda")
    reached = ctypes.c_uint64()
    hooks = G.get_test_hooks()
    try:
        G.set_test_hooks(noalloc_chunk_cap=cap)
        assert G.lib().gpma_bfs_noalloc(g.handle, 0, ctypes.c_void_p(levels.data_ptr()), ctypes.byref(reached),
                                        None) == 0
        overflows = G.get_test_hooks()["noalloc_overflows"]
    finally:
        G.set_test_hooks(**{k: hooks[k] for k in ("noalloc_chunk_cap",)})
    assert np.array_equal(levels.cpu().numpy(), want) and reached.value == n
    assert (overflows > 0) == (cap > 0)
    g.close()


def test_first_long_search_without_allocation_takes_no_memory():
    """In a process of its own: the second kernel is loaded by the first call, not
    by the first search that needs it."""
    code = """
import ctypes, numpy as np, torch
import gpma_bfs_gb300 as G
n = 300
u = np.arange(n - 1, dtype=np.uint64)
g = G.GPMA(n)
G.update_gpma(g, (u << np.uint64(32)) | (u + np.uint64(1)), np.ones(n - 1, np.uint8))
levels = torch.zeros(n, dtype=torch.int32, device="cuda")
def search(s):
    r = ctypes.c_uint64()
    assert G.lib().gpma_bfs_noalloc(g.handle, s, ctypes.c_void_p(levels.data_ptr()), ctypes.byref(r), None) == 0
    torch.cuda.synchronize()
    return r.value
assert search(n - 5) == 5
free = torch.cuda.mem_get_info()[0]
assert search(0) == n
assert torch.cuda.mem_get_info()[0] == free, free - torch.cuda.mem_get_info()[0]
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       cwd=Path(__file__).resolve().parent.parent)
    assert r.returncode == 0, r.stderr[-2000:]


def test_recorded_step(built_lib):
    n, src, dst, want = _hubs(100, 500)
    g = _graph(n, src, dst)
    k, v = np.array([5 << 32 | 7], np.uint64), np.zeros(1, np.uint8)  # a delete of nothing
    levels = np.zeros(n, np.uint32)
    with G.Step(g) as st:
        for _ in range(3):
            levels[:] = 9
            assert st.run(k, v, 0, levels) == n
            assert np.array_equal(levels, want)
        st.run(np.array([40 << 32 | 41], np.uint64), v, 0, levels)  # the chain ends at hub 40
        assert np.array_equal(levels, np.where(want <= 42, want, 0) * ~((want == 42) & (np.arange(n) == 41)))
    g.close()


def test_largest_items(built_lib):
    """An array of 2^27 slots and more, whose work items have four steps."""
    import torch

    h, leaves = 100, 600_000
    n = h * (leaves + 1)
    hub = torch.arange(h, device="cuda")
    keys = torch.cat([(hub[:-1] << 32) | hub[1:],
                      (hub.repeat_interleave(leaves) << 32) | (h + torch.arange(h * leaves, device="cuda"))])
    g = G.GPMA(n)
    G.update_gpma(g, keys, torch.ones(len(keys), dtype=torch.uint8, device="cuda"))
    assert g.get_size() >= 1 << 27
    levels = torch.zeros(n, dtype=torch.int32, device="cuda")
    _, reached = G.gpma_bfs(g, n, 0, 0, levels)
    assert reached == n
    assert torch.equal(levels[:h], (hub + 1).int())
    assert torch.equal(levels[h:].view(h, leaves), (hub + 2).int()[:, None].expand(h, leaves))
    g.close()
