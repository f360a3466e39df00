"""Which sweep a factor takes: along grid lines for the stencils' full patterns,
by levels or partitions for anything else, and by levels or partitions alone in
contexts that ask for them.  Without these checks a stencil that silently fell
back to the level-ordered sweep, or a pattern wrongly taken for a grid's, would
still agree with the level-ordered results bit for bit."""
import numpy as np
import pytest

from test_gpu_line_sweep import CASES, context, stencil

pytestmark = pytest.mark.gpu


def paths(P, M, prec):
    return [P.sweep_path(w, prec) for w in (M.LOWER, M.UPPER)]


@pytest.mark.parametrize("dims,box", CASES + [((300, 8, 8), True), ((97, 105, 9), True),
                                              ((64, 3, 30), True), ((12, 3, 8), False)])
@pytest.mark.parametrize("kind", ["ic0", "ilu0"])
def test_stencils_go_along_lines(M, dims, box, kind):
    rp, ci, v = stencil(dims, box)
    n = len(rp) - 1
    a, b = context(M), context(M, "ticket")
    try:
        A, B = M.Csr(a, rp, ci, v), M.Csr(b, rp, ci, v)
        P, Q = M.Pc(A, kind, M.FP32), M.Pc(B, kind, M.FP32)
        for prec in (M.FP64, M.FP32):
            assert paths(P, M, prec) == [M.SWEEP_LINES] * 2
            assert paths(Q, M, prec) == [M.SWEEP_LEVELS] * 2
        for which in (M.LOWER, M.UPPER):
            # the number of levels is known without an analysis; the levels after one
            info = P.factor_info(which)
            assert info == Q.factor_info(which)
            lev = P.levels(which)
            assert np.array_equal(lev, Q.levels(which))
            assert info[1] == lev.max() + 1 and P.factor_info(which) == info
        P.set_jacobi_sweeps(1)
        assert paths(P, M, M.FP64) == [M.SWEEP_JACOBI] * 2
        P.close(), Q.close(), A.close(), B.close()
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize("dims,box", [((16, 20), False), ((40, 37), True), ((6, 9, 11), False),
                                      ((6, 9, 11), True), ((20, 35, 9), False)])
@pytest.mark.parametrize("kind", ["ic0", "ilu0"])
def test_a_missing_entry_does_not(M, restate, dims, box, kind):
    rp, ci, v = stencil(dims, box, drop=int(np.prod(dims)) // 2)
    n = len(rp) - 1
    c = context(M)
    try:
        A = M.Csr(c, rp, ci, v)
        P = M.Pc(A, kind)
        assert M.SWEEP_LINES not in paths(P, M, M.FP64)
        r = M.uniform(n, 7)
        x, y = c.to_device(r), c.array(n)
        L, U = getattr(restate, kind)((n, rp, ci, v))
        P.sweep(M.LOWER, x, y)
        low = "lower_unit" if kind == "ilu0" else "lower_invdiag_last"
        assert np.array_equal(y.download(), restate.sweep(low, L, r))
        P.sweep(M.UPPER, x, y)
        assert np.array_equal(y.download(), restate.sweep("upper_invdiag_first", U, r))
        P.close(), A.close()
    finally:
        c.close()


@pytest.mark.parametrize("dims,path", [((200, 200), 1), ((30, 31, 32), 0), ((64, 64, 64), 0)])
def test_automatic_choice_without_a_grid(M, dims, path):
    # narrow levels and short rows: partitioned; wide levels: by levels
    rp, ci, v = stencil(dims, False, drop=int(np.prod(dims)) // 2)
    n = len(rp) - 1
    a, b = context(M), context(M, "ticket")
    try:
        A, B = M.Csr(a, rp, ci, v), M.Csr(b, rp, ci, v)
        P, Q = M.Pc(A, "ic0"), M.Pc(B, "ic0")
        r = M.uniform(n, 3)
        x, y, p, q = a.to_device(r), a.array(n), b.to_device(r), b.array(n)
        for which in (M.LOWER, M.UPPER):
            assert P.sweep_path(which) == path == P.sweep_kind(which)
            P.sweep(which, x, y)
            Q.sweep(which, p, q)
            assert np.array_equal(y.download(), q.download())
        P.close(), Q.close(), A.close(), B.close()
    finally:
        a.close()
        b.close()


def test_other_shapes_do_not(M, ctx):
    # a random graph, a tridiagonal matrix, lines shorter than eight rows
    for rp, ci, v in (M.random_graph(500, 6.0, 1e-2, 1)[1:], stencil((400,), False),
                      stencil((9, 9, 7), False), stencil((60, 7), True)):
        A = M.Csr(ctx, rp, ci, v)
        for kind in ("ic0", "ilu0"):
            P = M.Pc(A, kind)
            assert M.SWEEP_LINES not in paths(P, M, M.FP64)
            P.close()
        A.close()
