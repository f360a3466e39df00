"""CG's direction step split into a pass for p' and a plain product, taken by
stencil matrices of 2^20 rows and more, against the unfused iteration.

Both compute the same r, z, p and q element by element; only the order of the
dots' partial sums differs (<= 32 additions deep: 32 * 1.1e-16 of the sum of
magnitudes, ~4e-15).  A relative error e of alpha and beta moves the residual
history by about the iterations' count times a small factor of e: 1e-11 for
eight iterations leaves three digits of room.
"""
import os

import numpy as np
import pytest

SIZES = [(1 << 20, "2d", 1024, 1024), (1024 * 1031, "2d", 1031, 1024), (102 ** 3, "3d", 102, 0)]


def _matrix(M, ctx, kind, a, b):
    return M.Csr.laplacian2d(ctx, a, b) if kind == "2d" else M.Csr.laplacian3d(ctx, a)


@pytest.mark.gpu
@pytest.mark.parametrize("n,kind,a,b", SIZES)
@pytest.mark.parametrize("sweeps", [1, 2])
def test_history_matches_unfused(M, ctx, n, kind, a, b, sweeps):
    rhs = M.uniform(n, 5)
    hist = {}
    for fused in ("1", "0"):
        old = os.environ.get("MTLGPU_CG_FUSED")
        os.environ["MTLGPU_CG_FUSED"] = fused
        try:
            A = _matrix(M, ctx, kind, a, b)
            P = M.Pc(A, "ic0")
            P.set_jacobi_sweeps(sweeps)
            x, db = ctx.to_device(np.zeros(n)), ctx.to_device(rhs)
            _, _, h = M.solve("cg", A, P, x, db, rtol=1e-14, max_iter=8)
            hist[fused] = (h, x.download())
            P.close()
            A.close()
        finally:
            if old is None:
                os.environ.pop("MTLGPU_CG_FUSED", None)
            else:
                os.environ["MTLGPU_CG_FUSED"] = old
    h1, h0 = hist["1"][0], hist["0"][0]
    assert len(h1) == len(h0) == 9
    assert np.all(h0 > 0) and np.all(np.abs(h1 - h0) <= 1e-11 * h0)
    assert np.linalg.norm(hist["1"][1] - hist["0"][1]) <= 1e-11 * np.linalg.norm(hist["0"][1])


@pytest.mark.gpu
def test_mixed_solve_reaches_its_tolerance(M, ctx):
    n = 102 ** 3
    A = M.Csr.laplacian3d(ctx, 102)
    P = M.Pc(A, "ic0", M.FP32)
    P.set_jacobi_sweeps(1)
    b = M.uniform(n, 6)
    x, db = ctx.to_device(np.zeros(n)), ctx.to_device(b)
    st, res, _ = M.solve("cg", A, P, x, db, rtol=1e-9, max_iter=4000, mode=M.SOLVE_MIXED,
                         inner_rtol=1e-5)
    assert st == M.OK
    g = x.download().reshape(102, 102, 102)
    ax = 6.0 * g
    for d in range(3):
        lo = tuple(slice(0, -1) if k == d else slice(None) for k in range(3))
        hi = tuple(slice(1, None) if k == d else slice(None) for k in range(3))
        ax[lo] -= g[hi]
        ax[hi] -= g[lo]
    # rounding of A x itself: a few 1e-16 of ||A|| ||x||, far below 1e-10 ||b||
    assert np.linalg.norm(ax.ravel() - b) <= 1.1e-9 * np.linalg.norm(b)
