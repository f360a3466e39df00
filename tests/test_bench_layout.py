"""The benchmark's bytes per entry and row follow the library's choice of layout."""
import os
import sys

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


def test_layout_bytes(M, monkeypatch):
    import bench
    monkeypatch.delenv("MTLGPU_SELL_INDEX", raising=False)
    assert bench.layout_bytes(*M.laplacian3d(12)[1:3]) == (0, 1)
    assert bench.layout_bytes(*M.convdiff27(12, 2)[1:3]) == (0, 4)
    # rows of very different length: CSR-stream
    assert bench.layout_bytes(*M.random_graph(900, 6.0, 1e-2, 1)[1:3]) == (4, 4)
    # even rows, an offset of their own each: SELL-32
    n = 64
    ci = np.stack([np.arange(n), n + (np.arange(n) * 7) % 61]).T
    rp = np.arange(0, 2 * n + 1, 2)
    assert bench.layout_bytes(rp, ci.ravel()) == (2, 4 / 32)
    monkeypatch.setenv("MTLGPU_SELL_INDEX", "32")
    assert bench.layout_bytes(*M.laplacian3d(12)[1:3]) == (4, 4 / 32)
