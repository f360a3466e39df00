"""Which layout a matrix's products read: the grid layout for at most 32 distinct
offsets column - row, where padding every row to all of them adds at most a
quarter and padding to slices of 32 rows a fifth; SELL-32 for other rows of even
length; CSR-stream for the rest.  Products agree bit for bit whatever is chosen, so
only this tells whether the grid kernels ran."""
import numpy as np
import pytest

from test_gpu_grid_layout import CASES, offsets_matrix, sym

pytestmark = pytest.mark.gpu


def expected(M, A):
    n, rp, ci, _ = A
    ln = np.diff(rp)
    padded = np.pad(ln, (0, -n % 32)).reshape(-1, 32).max(1).sum() * 32
    if padded > 1.2 * len(ci):
        return M.LAYOUT_STREAM
    w = len(np.unique(ci - np.repeat(np.arange(n), ln)))
    return M.LAYOUT_GRID if w <= 32 and w * n <= 1.25 * len(ci) else M.LAYOUT_SELL


def test_of_the_equality_tests(M, ctx):
    got = []
    for n, offs, drop in CASES:
        A = offsets_matrix(n, offs, drop, n)
        dA = M.Csr(ctx, *A[1:])
        got.append(dA.layout())
        assert got[-1] == expected(M, A), (n, offs, drop)
        dA.close()
    # 12 of the 19 are on the grid layout (offsets near the number of rows leave too
    # many rows without them); the one with 33 offsets is not
    assert got.count(M.LAYOUT_GRID) == 12
    n, offs, _ = next(c for c in CASES if len(c[1]) == 33)
    assert got[[c[1] for c in CASES].index(offs)] == M.LAYOUT_SELL


@pytest.mark.parametrize("W", range(1, 34))
def test_by_number_of_offsets(M, ctx, W):
    offs = [0] + [s * (7 * i + 3) for i in range((W - 1) // 2) for s in (1, -1)]
    offs += [331] if W % 2 == 0 else []
    dA = M.Csr(ctx, *offsets_matrix(4000, offs, 0.0, W)[1:])
    assert dA.layout() == (M.LAYOUT_GRID if W <= 32 else M.LAYOUT_SELL)
    dA.close()


def test_of_other_matrices(M, ctx, monkeypatch):
    lap = M.laplacian3d(20)
    for A, want in ((lap, M.LAYOUT_GRID), (M.convdiff27(20, 2), M.LAYOUT_GRID),
                    (M.random_graph(900, 6.0, 1e-2, 1), M.LAYOUT_STREAM),
                    (offsets_matrix(3000, sym(31) + [200, 201], 0.0, 1), M.LAYOUT_SELL)):
        dA = M.Csr(ctx, *A[1:])
        assert dA.layout() == want
        dA.close()
    # one row with an offset of its own, which no sample need find
    n, rp, ci, v = offsets_matrix(200000, sym(7), 0.0, 1)
    at = rp[77777] + int(np.searchsorted(ci[rp[77777]:rp[77778]], 77777 + 155))
    rp2 = rp + (np.arange(n + 1) > 77777)
    dA = M.Csr(ctx, rp2, np.insert(ci, at, 77777 + 155), np.insert(v, at, 0.5))
    assert dA.layout() == M.LAYOUT_SELL
    dA.close()
    dA = M.Csr(ctx, *lap[1:])
    dA.autotune()
    assert dA.layout() in (M.LAYOUT_GRID, M.LAYOUT_STREAM)
    dA.close()
    monkeypatch.setenv("MTLGPU_SELL_INDEX", "32")
    dA = M.Csr(ctx, *lap[1:])
    assert dA.layout() == M.LAYOUT_SELL
    dA.close()
