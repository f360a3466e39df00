"""The spin limit bounds one wait of a sweep along grid lines, not the polls of
the whole sweep: lines of 100,000 rows (two tiles, so that one waits for the
other) are swept with a limit that every single wait keeps far below and the
sweep's polls together exceed many times over.  A step of the sweep takes ~60 ns,
so it runs for 6 ms; a loader polls every ~70 ns (90,000 polls) and the second
tile's fetch every ~0.5 us (12,000); the limit of 4,096 polls is 150 us or more."""
import numpy as np
import pytest

from test_gpu_line_sweep import context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float64, np.float32])
def test_limit_is_of_one_wait(M, dt):
    c = context(M)
    try:
        A = M.Csr.laplacian2d(c, 40, 100000)
        P = M.Pc(A, "ic0", M.FP32)
        x, y = c.to_device(np.ones(A.n, dt)), c.array(A.n, dt)
        want = {}
        for which in (M.LOWER, M.UPPER):
            P.sweep(which, x, y)
            want[which] = y.download()
        c.set_spin_limit(4096)
        for which in (M.LOWER, M.UPPER):
            P.sweep(which, x, y)
            assert np.array_equal(y.download(), want[which])
        P.close(), A.close()
    finally:
        c.close()


@pytest.mark.parametrize("limit", [1, 16, 300])
@pytest.mark.parametrize("grid", ["lines", "cube"])
def test_a_wait_that_runs_out_leaves_the_context_usable(M, limit, grid):
    """Lines of many more stages than a block holds: a warp that gives up stops its
    loader, and the block ends once its copies have landed."""
    c = context(M)
    try:
        A = M.Csr.laplacian2d(c, 40, 20000) if grid == "lines" else M.Csr.laplacian3d(c, 100)
        P = M.Pc(A, "ic0", M.FP32)
        for dt in (np.float64, np.float32):
            x, y = c.to_device(M.uniform(A.n, 3).astype(dt)), c.array(A.n, dt)
            for which in (M.LOWER, M.UPPER):
                P.sweep(which, x, y)
                want = y.download()
                c.set_spin_limit(limit)
                for _ in range(4):
                    try:
                        P.sweep(which, x, y)
                    except M.MtlgpuError as e:
                        assert e.status == M.TIMEOUT
                c.set_spin_limit(1 << 26)
                P.sweep(which, x, y)
                assert np.array_equal(y.download(), want)
        P.close(), A.close()
    finally:
        c.close()
