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


def _planes(planes, lines, length):
    """The 27-point stencil on planes x lines x length by repeating an inner plane."""
    rp, ci, v = stencil((5, lines, length), True)
    m = lines * length
    cnt = np.diff(rp)
    lo, hi = rp[2 * m], rp[3 * m]
    k = planes - 4
    inner = (ci[lo:hi][None, :] + (m * np.arange(k))[:, None]).ravel()
    count = np.concatenate([cnt[:2 * m], np.tile(cnt[2 * m:3 * m], k), cnt[3 * m:]])
    cols = np.concatenate([ci[:lo], inner, ci[hi:] + m * (planes - 5)])
    vals = np.concatenate([v[:lo], np.tile(v[lo:hi], k), v[hi:]])
    return (np.concatenate([[0], np.cumsum(count)]).astype(np.int32), cols.astype(np.int32), vals)


def test_planes_repeat_the_stencil():
    for a, b in zip(_planes(9, 3, 8)[:2], stencil((9, 3, 8), True)[:2]):
        assert np.array_equal(a, b)


def test_records_of_thin_grids_are_bounded(M):
    # 2.6 M rows in planes of three lines of eight: a factor's records would take
    # 21 times its rows' 340 MB, more than a 32nd of the device
    rp, ci, v = _planes(110000, 3, 8)
    n = len(rp) - 1
    import torch
    c, d = context(M), context(M, "ticket")
    try:
        A, B = M.Csr(c, rp, ci, v), M.Csr(d, rp, ci, v)
        Q = M.Pc(B, "ic0")
        q, w = d.to_device(M.uniform(n, 2)), d.array(n)
        Q.apply(q, w)
        before = torch.cuda.mem_get_info(0)[0]
        P = M.Pc(A, "ic0")
        x, y = c.to_device(M.uniform(n, 2)), c.array(n)
        P.apply(x, y)
        assert before - torch.cuda.mem_get_info(0)[0] < 4 << 30
        assert np.array_equal(y.download(), w.download())
        P.close(), Q.close(), A.close(), B.close()
    finally:
        c.close()
        d.close()
