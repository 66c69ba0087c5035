"""Source lists in plain host memory are read after the work that is on the stream
before the search: a host function on the stream writes them a while later."""
import ctypes
import time

import numpy as np
import pytest

import gpma_bfs_gb300 as G

pytestmark = pytest.mark.gpu


def _written_later(stream, array, values):
    """Enqueues a host function that waits and then writes the array; returns what must stay alive."""
    def write(_):
        time.sleep(0.1)
        array[:] = values

    fn = ctypes.CFUNCTYPE(None, ctypes.c_void_p)(write)
    rt = ctypes.CDLL("libcudart.so.13")
    assert rt.cudaLaunchHostFunc(ctypes.c_void_p(stream.cuda_stream), fn, None) == 0
    return fn


def test_sources_are_read_in_stream_order(built_lib):
    import torch

    n = 2000
    u = np.arange(n - 1, dtype=np.uint64)
    g = G.GPMA(n)  # a path: node s reaches n - s nodes
    G.update_gpma(g, (u << np.uint64(32)) | (u + np.uint64(1)), np.ones(n - 1, np.uint8))
    s = torch.cuda.Stream()
    late = np.array([1500, 1700], np.uint32)
    src = np.zeros(2, np.uint32)
    keep = _written_later(s, src, late)
    _, reached = G.gpma_bfs_multi(g, src, stream=s)
    assert reached.tolist() == [500, 300]
    # many graphs, through the C call: Batch.bfs_multi copies the lists first
    src = np.zeros(2, np.uint32)
    keep = _written_later(s, src, late)
    b = G.Batch()
    hs = (ctypes.c_void_p * 1)(g.handle.value)
    sp, ns = (ctypes.c_void_p * 1)(src.ctypes.data), (ctypes.c_uint32 * 1)(2)
    reached = np.zeros(2, np.uint64)
    assert G.lib().gpma_batch_bfs_multi(b._h, hs, sp, ns, 1, None, reached.ctypes.data_as(ctypes.c_void_p),
                                        ctypes.c_void_p(s.cuda_stream)) == 0
    assert reached.tolist() == [500, 300]
    torch.cuda.synchronize()
    del keep
    b.close()
    g.close()
