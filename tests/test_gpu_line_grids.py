"""Sweeps along the lines of grids that are much longer one way than the other:
27-point factors, whose lines are shifted by one per plane, against the
level-ordered sweep (MTLGPU_SWEEP=ticket), bit for bit, and the device memory
they take, which follows the rows and not the square of the planes."""
import numpy as np
import pytest

from test_gpu_line_sweep import context, stencil

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(300, 8, 8), (301, 9, 11), (150, 2, 8), (64, 3, 30), (7, 90, 8),
                                  (97, 105, 9)])
@pytest.mark.parametrize("kind", ["ic0", "ilu0"])
def test_long_grids_equal_level_sweep(M, dims, kind):
    rp, ci, v = stencil(dims, True)
    n = len(rp) - 1
    a, b = context(M), context(M, "ticket")
    try:
        A, B = M.Csr(a, rp, ci, v), M.Csr(b, rp, ci, v)
        P, Q = M.Pc(A, kind, M.FP32), M.Pc(B, kind, M.FP32)
        for which in (M.LOWER, M.UPPER):
            assert all(np.array_equal(x, y)
                       for x, y in zip(P.factor(which)[1:], Q.factor(which)[1:]))
            for dt in (np.float64, np.float32):
                r = M.uniform(n, 5).astype(dt)
                x, y = a.to_device(r), a.array(n, dt)
                p, q = b.to_device(r), b.array(n, dt)
                P.sweep(which, x, y)
                Q.sweep(which, p, q)
                assert np.array_equal(y.download(), q.download()), (dt, which)
        P.close(), Q.close(), A.close(), B.close()
    finally:
        a.close()
        b.close()


def test_memory_of_a_long_grid(M):
    # 128,000 rows: a factor's records take 16 MB, with their padding twelve
    # times that; tiles of the sheared bounding box took 16 GB
    import torch
    rp, ci, v = stencil((2000, 8, 8), True)
    n = len(rp) - 1
    c = context(M)
    try:
        A = M.Csr(c, rp, ci, v)
        before = torch.cuda.mem_get_info(0)[0]
        P = M.Pc(A, "ic0")
        x, y = c.to_device(M.uniform(n, 2)), c.array(n)
        P.apply(x, y)
        assert before - torch.cuda.mem_get_info(0)[0] < 1 << 30
        P.close(), A.close()
    finally:
        c.close()
