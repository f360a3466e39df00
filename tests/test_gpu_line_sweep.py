"""Sweeps along grid lines (the default for factors with a grid stencil's
pattern) against the level-ordered sweep (MTLGPU_SWEEP=ticket): both follow the
reference's per-row operation order (lower_trisolve.hpp:173-209,
upper_trisolve.hpp:160-176) with separately rounded operations, so the results
are equal bit for bit.  Sizes around the tiles (patches of 4 x 8 or 32 lines,
tiles of 16 x 8, blocks of 4 rows), the shortest lines, grids whose sides
differ, and patterns that only resemble a grid's."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def context(M, mode=None):
    old = os.environ.pop("MTLGPU_SWEEP", None)
    if mode:
        os.environ["MTLGPU_SWEEP"] = mode
    try:
        return M.Context(0)
    finally:
        os.environ.pop("MTLGPU_SWEEP", None)
        if old is not None:
            os.environ["MTLGPU_SWEEP"] = old


def stencil(dims, box, seed=1, drop=None):
    """CSR of a grid stencil with random values, rows in natural order: the
    nearest neighbours, or (box) all of the surrounding box; `drop` removes one
    off-diagonal entry pair of the given row and its successor."""
    g = np.random.default_rng(seed)
    idx = np.arange(int(np.prod(dims))).reshape(dims)
    r, c = [], []
    nd = len(dims)
    for off in np.ndindex(*(3,) * nd):
        o = np.array(off) - 1
        if not box and np.abs(o).sum() > 1:
            continue
        src = tuple(slice(max(0, -x), d - max(0, x)) for x, d in zip(o, dims))
        dst = tuple(slice(max(0, x), d - max(0, -x)) for x, d in zip(o, dims))
        r.append(idx[src].ravel())
        c.append(idx[dst].ravel())
    r, c = np.concatenate(r), np.concatenate(c)
    if drop is not None:
        keep = ~(((r == drop) & (c == drop + 1)) | ((r == drop + 1) & (c == drop)))
        r, c = r[keep], c[keep]
    order = np.lexsort((c, r))
    r, c = r[order], c[order]
    n = idx.size
    v = g.uniform(-1.0, -0.2, len(r))
    v[r == c] = 30.0 + g.uniform(0, 1, n)
    rp = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(r, minlength=n), out=rp[1:])
    return rp, c.astype(np.int32), v


CASES = [((8, 8), False), ((9, 31), False), ((32, 33), False), ((65, 8), False), ((3, 200), False),
         ((40, 37), True), ((9, 8), True), ((70, 64), True),
         ((4, 8, 8), False), ((5, 9, 11), False), ((17, 16, 13), False), ((2, 3, 40), False),
         ((33, 8, 10), False), ((20, 35, 9), False),
         ((4, 8, 8), True), ((5, 9, 11), True), ((17, 16, 13), True), ((2, 3, 40), True),
         ((33, 9, 8), True), ((18, 33, 10), True),
         # more tiles of 8 x 8 lines than SMs: the 16 x 8 form
         ((97, 105, 8), False), ((75, 101, 9), True)]


@pytest.mark.parametrize("dims,box", CASES)
@pytest.mark.parametrize("kind", ["ic0", "ilu0"])
def test_line_sweep_equals_level_sweep(M, dims, box, kind):
    rp, ci, v = stencil(dims, box)
    n = len(rp) - 1
    a, b = context(M), context(M, "ticket")
    try:
        A, B = M.Csr(a, rp, ci, v), M.Csr(b, rp, ci, v)
        P, Q = M.Pc(A, kind, M.FP32), M.Pc(B, kind, M.FP32)
        for dt in (np.float64, np.float32):
            r = M.uniform(n, 5).astype(dt)
            x, y = a.to_device(r), a.array(n, dt)
            p, q = b.to_device(r), b.array(n, dt)
            for which in (M.LOWER, M.UPPER):
                for _ in range(2):          # the tile counter is ready again
                    P.sweep(which, x, y)
                Q.sweep(which, p, q)
                assert np.array_equal(y.download(), q.download()), (dt, which)
        r = M.uniform(n, 6)
        x, y = a.to_device(r), a.array(n)
        p, q = b.to_device(r), b.array(n)
        for f in ("apply", "adjoint_apply"):
            getattr(P, f)(x, y)
            getattr(Q, f)(p, q)
            assert np.array_equal(y.download(), q.download()), f
        P.close(), Q.close(), A.close(), B.close()
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize("dims,box", [((16, 20), False), ((6, 9, 11), False), ((6, 9, 11), True)])
def test_a_missing_entry_keeps_the_level_sweep_result(M, restate, dims, box):
    # one coupling inside the grid is absent: not the full stencil's pattern
    rp, ci, v = stencil(dims, box, drop=int(np.prod(dims)) // 2)
    n = len(rp) - 1
    c = context(M)
    try:
        A = M.Csr(c, rp, ci, v)
        P = M.Pc(A, "ilu0")
        r = M.uniform(n, 7)
        x, y = c.to_device(r), c.array(n)
        L, U = restate.ilu0((n, rp, ci, v))
        P.sweep(M.LOWER, x, y)
        assert np.array_equal(y.download(), restate.sweep("lower_unit", L, r))
        P.sweep(M.UPPER, x, y)
        assert np.array_equal(y.download(), restate.sweep("upper_invdiag_first", U, r))
        P.close(), A.close()
    finally:
        c.close()


def test_line_sweep_with_nonfinite_values(M):
    # inf and NaN right-hand sides travel as in the level-ordered sweep
    rp, ci, v = stencil((9, 10, 12), False)
    n = len(rp) - 1
    a, b = context(M), context(M, "ticket")
    try:
        A, B = M.Csr(a, rp, ci, v), M.Csr(b, rp, ci, v)
        P, Q = M.Pc(A, "ic0"), M.Pc(B, "ic0")
        r = M.uniform(n, 8)
        r[n // 3], r[n // 2], r[5] = np.inf, np.nan, -0.0
        x, y = a.to_device(r), a.array(n)
        p, q = b.to_device(r), b.array(n)
        for which in (M.LOWER, M.UPPER):
            P.sweep(which, x, y)
            Q.sweep(which, p, q)
            assert np.array_equal(y.download(), q.download(), equal_nan=True)
        P.close(), Q.close(), A.close(), B.close()
    finally:
        a.close()
        b.close()


def test_line_sweep_timeout_leaves_the_context_usable(M):
    c = context(M)
    try:
        A = M.Csr.laplacian3d(c, 24)
        P = M.Pc(A, "ic0")
        x, y = c.to_device(np.ones(A.n)), c.array(A.n)
        P.apply(x, y)
        want = y.download()
        c.set_spin_limit(1)
        with pytest.raises(M.MtlgpuError) as e:
            P.apply(x, y)
        assert e.value.status == M.TIMEOUT
        c.set_spin_limit(1 << 22)
        P.apply(x, y)
        assert np.array_equal(y.download(), want)
        P.close(), A.close()
    finally:
        c.close()
