"""The first array of a new graph, written directly from the row numbers,
against the oracle's update of the initial 4-slot array by all guards: tiny
row counts where the root's integer bounds drop the guards, powers of two and
their neighbours (density edges of a size), and ragged sizes."""
import numpy as np
import pytest

from oracle.oracle import OracleGPMA
from replay import GpuAdapter

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [0, 1, 2, 3, 4, 5, 6, 7, 11, 12, 13, 31, 105, 106, 1023, 1717, 1718, 1719, 65536, 99991])
def test_new_graph_equals_oracle(built_lib, rows):
    gpu, orc = GpuAdapter(rows), OracleGPMA(rows, threads=2)
    assert gpu.geometry() == orc.geometry()
    for name, a, b in zip(("keys", "values", "row_offset"), gpu.export_layout(), orc.export_layout()):
        assert np.array_equal(a, b), name
    assert gpu.g.validate() == 0 and gpu.g.stats()["updates"] == 0
    if rows > 1:
        k = np.array([(rows - 1) << 32, 1, 1 << 32], np.uint64)
        v = np.ones(3, np.uint8)
        gpu.update(k, v)
        orc.update(k, v)
        assert all(np.array_equal(a, b) for a, b in zip(gpu.export_layout(), orc.export_layout()))
    gpu.close()


def test_new_graph_with_bulk_sized_guards(built_lib):
    """From 5M rows on the guards' insertion is the bulk rebuild, whose gaps hold key 0."""
    rows = 5_000_000
    gpu, orc = GpuAdapter(rows), OracleGPMA(rows, threads=8)
    assert gpu.geometry() == orc.geometry()
    assert all(np.array_equal(a, b) for a, b in zip(gpu.export_layout(), orc.export_layout()))
    assert gpu.g.validate() == 0
    gpu.close()
