"""Every number of offsets the grid layout takes, 1 to 32 (those without a kernel of
their own in chunks of 8 and a remainder of 1 to 7), against the 32-bit index
layout (MTLGPU_SELL_INDEX=32) and the oracle: products and Jacobi-applied factors bit
for bit, CG and BiCGSTAB (whose dots are grouped differently) to 1e-8."""
import numpy as np
import pytest

from test_gpu_grid_layout import offsets_matrix
from test_gpu_layout_choice import expected

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", range(1, 33))
def test_width(M, restate, monkeypatch, W):
    k = (W - 1) // 2
    offs = [0] + [s * (7 * i + 3) for i in range(k) for s in (1, -1)] + ([331] if W % 2 == 0 else [])
    n = 2003
    A = offsets_matrix(n, offs, 0.0, W)
    if W % 2:                   # symmetric values, for CG
        r = np.repeat(np.arange(n), np.diff(A[1]))
        lo, hi = np.minimum(r, A[2]), np.maximum(r, A[2])
        A[3][r != A[2]] = np.cos(0.7 * lo + 1.3 * hi)[r != A[2]]
    x64, x32 = M.uniform(n, 5), M.uniform(n, 6).astype(np.float32)
    out = {}
    for layout in ("grid", "32"):
        if layout == "32":
            monkeypatch.setenv("MTLGPU_SELL_INDEX", "32")
        c = M.Context(0)
        dA = M.Csr(c, *A[1:])
        y64, y32 = c.array(n), c.array(n, np.float32)
        a64, a32 = c.to_device(x64), c.to_device(x32)
        res = []
        dA.spmv(a64, y64)
        dA.spmv_f32(a32, y32)
        res += [y64.download(), y32.download()]
        assert np.array_equal(res[0], restate.spmv(A, x64))
        P = M.Pc(dA, "ilu0", M.FP32)
        P.set_jacobi_sweeps(2)
        P.apply(a64, y64)
        P.apply_f32(a32, y32)
        res += [y64.download(), y32.download()]
        for method in ("bicgstab", "cg") if W % 2 else ("bicgstab",):
            for mode in (M.SOLVE_FP64, M.SOLVE_MIXED):
                x = c.to_device(np.zeros(n))
                st, _, _ = M.solve(method, dA, P, x, a64, rtol=1e-10, max_iter=500, mode=mode)
                assert st == M.OK
                res.append(x.download())
        out[layout] = res
        P.close(), dA.close(), c.close()
    for j, (g, i) in enumerate(zip(out["grid"], out["32"])):
        if j < 4:
            assert np.array_equal(g, i), j
        else:
            assert np.linalg.norm(g - i) <= 1e-8 * np.linalg.norm(i), j


@pytest.mark.parametrize("n", [8, 31, 32, 33, 64, 127, 128, 129, 160, 255, 256, 257, 383, 384,
                               385, 1000])
@pytest.mark.parametrize("offs", [[0], [0, 1], [-2, 0], [0, 1, -1], [0, 1, -1, 2, -2]])
def test_row_counts(M, ctx, restate, n, offs):
    # around warps and slices of 128 rows; a vector off the 16-byte grid
    A = offsets_matrix(n, offs, 0.0, n)
    dA = M.Csr(ctx, *A[1:])
    assert dA.layout() == expected(M, A)
    x = M.uniform(n, 3)
    for shift in (0, 1):
        a, y = ctx.to_device(np.concatenate([np.zeros(shift), x])), ctx.array(n + shift)

        class View:
            def __init__(self, v):
                self.n, self.ptr = n, M.C.c_void_p(v.ptr.value + 8 * shift)
        dA.spmv(View(a), View(y))
        assert np.array_equal(y.download()[shift:], restate.spmv(A, x))
    dA.close()
