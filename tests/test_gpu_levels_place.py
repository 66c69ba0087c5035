"""Levels in every kind of memory a caller may pass, also several kinds in one
call of many graphs: device (aligned, and one byte off), managed, page-locked and
plain host memory, and none."""
import ctypes

import numpy as np
import pytest

import gpma_bfs_gb300 as G

pytestmark = pytest.mark.gpu

KINDS = ["device", "off", "managed", "pinned", "plain", "none"]


class Levels:
    """count uint32 of one kind of memory, filled with 7."""

    def __init__(self, kind, count):
        import torch

        self.kind, self.n, self.ptr = kind, 4 * count, None
        fill = np.full(count, 7, np.uint32).view(np.uint8)
        if kind == "managed":
            self.rt = ctypes.CDLL("libcudart.so.13")
            p = ctypes.c_void_p()
            assert self.rt.cudaMallocManaged(ctypes.byref(p), ctypes.c_size_t(self.n), 1) == 0
            self.ptr = p.value
            ctypes.memmove(self.ptr, fill.ctypes.data, self.n)
        elif kind == "plain":
            self.a = fill.copy()
            self.ptr = self.a.ctypes.data
        elif kind != "none":
            off = 1 if kind == "off" else 0
            self.t = torch.zeros(self.n + off, dtype=torch.uint8)
            self.t[off:] = torch.from_numpy(fill.copy())
            self.t = self.t.pin_memory() if kind == "pinned" else self.t.cuda()
            self.ptr = self.t.data_ptr() + off

    def read(self):
        if self.kind == "plain":
            b = self.a
        elif self.kind == "managed":
            b = np.ctypeslib.as_array((ctypes.c_uint8 * self.n).from_address(self.ptr)).copy()
            self.rt.cudaFree(ctypes.c_void_p(self.ptr))
        else:
            b = self.t.cpu().numpy()[self.t.numel() - self.n:].copy()
        return b.view(np.uint32)


def _graph(n, m, seed):
    rng = np.random.default_rng(seed)
    k = (rng.integers(0, n, m).astype(np.uint64) << np.uint64(32)) | rng.integers(0, n, m).astype(np.uint64)
    g = G.GPMA(n)
    G.update_gpma(g, np.unique(k), np.ones(len(np.unique(k)), np.uint8))
    return g


def _ok(status):
    assert status == 0, G.lib().gpma_last_error()


@pytest.mark.parametrize("kind", KINDS[:-1])
def test_single_graph_calls(built_lib, kind):
    n = 5003
    g = _graph(n, 20000, 3)
    want, _ = G.gpma_bfs(g, n, 0, 11)
    lv = Levels(kind, n)
    _ok(G.lib().gpma_bfs(g.handle, 11, ctypes.c_void_p(lv.ptr), None, None))
    assert np.array_equal(lv.read(), want)
    src = np.array([11, 5, 11, 4000], np.uint32)
    want4, _ = G.gpma_bfs_multi(g, src)
    lv = Levels(kind, 4 * n)
    _ok(G.lib().gpma_bfs_multi(g.handle, src.ctypes.data_as(ctypes.c_void_p), 4, ctypes.c_void_p(lv.ptr), None, None))
    assert np.array_equal(lv.read().reshape(4, n), want4)
    k = np.array([(11 << 32) | 4999, (4999 << 32) | 5000], np.uint64)
    v = np.ones(2, np.uint8)
    with G.Step(g) as st:
        for _ in range(2):  # recorded, then replayed
            lv = Levels(kind, n)
            r = ctypes.c_uint64()
            _ok(G.lib().gpma_step_run(st.handle, k.ctypes.data_as(ctypes.c_void_p),
                                      v.ctypes.data_as(ctypes.c_void_p), ctypes.c_uint64(2), 11,
                                      ctypes.c_void_p(lv.ptr), ctypes.byref(r), None))
            want, reached = G.gpma_bfs(g, n, 0, 11)
            assert r.value == reached and np.array_equal(lv.read(), want)
    g.close()


def test_several_kinds_in_one_call(built_lib):
    gs = [_graph(900 + 101 * i, 4000, i) for i in range(len(KINDS))]
    srcs = [np.arange(1, 2 + 9 * i, dtype=np.uint32) for i in range(len(KINDS))]  # 1 to 46 sources
    b = G.Batch()
    want, want_reached = b.bfs_multi(gs, srcs, levels=True)
    lv = [Levels(kind, len(s) * g.row_num) for kind, s, g in zip(KINDS, srcs, gs)]
    k = len(gs)
    hs = (ctypes.c_void_p * k)(*[g.handle.value for g in gs])
    sp = (ctypes.c_void_p * k)(*[s.ctypes.data for s in srcs])
    ns = (ctypes.c_uint32 * k)(*[len(s) for s in srcs])
    lp = (ctypes.c_void_p * k)(*[x.ptr for x in lv])
    reached = np.zeros(sum(len(s) for s in srcs), np.uint64)
    _ok(G.lib().gpma_batch_bfs_multi(b._h, hs, sp, ns, k, lp, reached.ctypes.data_as(ctypes.c_void_p), None))
    assert np.array_equal(reached, np.concatenate(want_reached))
    for kind, x, w in zip(KINDS, lv, want):
        if kind != "none":
            assert np.array_equal(x.read().reshape(w.shape), w), kind
    b.close()
    for g in gs:
        g.close()
