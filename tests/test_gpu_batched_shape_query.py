"""The shape that the batched autotuner keeps can be read back whole, and asked for
again by MTLGPU_BATCH_SHAPE with the same bits (the shape fixes the order of every
sum)."""
import numpy as np
import pytest


@pytest.mark.gpu
def test_tuned_shape_reads_back(M, ctx, monkeypatch):
    _, (n, rp, ci, v, off) = M.graph_batch(12, 500, 6000, 8.0, 32.0, 1e-2, seed=6)
    b = ctx.to_device(M.normal(n, 4))
    x = ctx.to_device(np.zeros(n))
    A = M.Csr(ctx, rp, ci, v)
    P = M.Pc(A, "diagonal")
    assert M.batched_shape(A) == (0, 0, 0, 0)
    choice = M.batched_autotune(A, P, off, x, b, rtol=1e-8, max_iter=2000)
    ctas, lanes, threads, rows = M.batched_shape(A)
    assert choice == 1000 * rows + 100 * ctas + lanes
    assert threads in ((256, 512, 1024) if lanes in (1, 8) else (256,))
    st, _ = M.solve_batched(A, P, off, x, b, rtol=1e-8, max_iter=2000)
    assert st == M.OK
    tuned = x.download()
    B = M.Csr(ctx, rp, ci, v)
    Q = M.Pc(B, "diagonal")
    monkeypatch.setenv("MTLGPU_BATCH_SHAPE", "%d,%d,%d,%d" % (ctas, lanes, rows, threads))
    x.upload(np.zeros(n))
    st, _ = M.solve_batched(B, Q, off, x, b, rtol=1e-8, max_iter=2000)
    assert st == M.OK and np.array_equal(x.download(), tuned)
    for h in (P, Q, A, B):
        h.close()
