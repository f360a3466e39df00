"""mtlgpu_pc_apply_f32 is asynchronous: its first call may be recorded into a
caller's CUDA graph.  The graph and the calls after it give the results of the
same preconditioner in an ordinary context, for factors swept along grid lines,
by levels and by Jacobi iterations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", ["lap2d", "lap3d", "cd27", "graph"])
@pytest.mark.parametrize("kind", ["ic0", "ilu0"])
@pytest.mark.parametrize("jacobi", [0, 2])
def test_first_apply_inside_a_capture(M, ctx, grid, kind, jacobi):
    import torch
    H = {"lap2d": lambda: M.laplacian2d(40, 37), "lap3d": lambda: M.laplacian3d(17),
         "cd27": lambda: M.convdiff27(13, 2), "graph": lambda: M.random_graph(900, 6.0, 1e-2, 1)}
    n, rp, ci, v = H[grid]()
    r, r2 = M.uniform(n, 3).astype(np.float32), M.uniform(n, 4).astype(np.float32)
    A0 = M.Csr(ctx, rp, ci, v)
    P0 = M.Pc(A0, kind, M.FP32)
    P0.set_jacobi_sweeps(jacobi)
    want = []
    for w in (r, r2):
        z0 = ctx.array(n, np.float32)
        P0.apply_f32(ctx.to_device(w), z0)
        ctx.synchronize()
        want.append(z0.download())
    s = torch.cuda.Stream()
    c = M.Context(0, stream=s.cuda_stream)
    try:
        A = M.Csr(c, rp, ci, v)
        P = M.Pc(A, kind, M.FP32)
        P.set_jacobi_sweeps(jacobi)
        x, z = c.to_device(r), c.array(n, np.float32)
        c.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            P.apply_f32(x, z)
        for w, k in ((r, 0), (r2, 1), (r, 0)):
            x.upload(w)
            with torch.cuda.stream(s):
                g.replay()
            c.synchronize()
            assert np.array_equal(z.download(), want[k])
        P.apply_f32(x, z)
        c.synchronize()
        assert np.array_equal(z.download(), want[0])
        del g
        P.close(), A.close()
    finally:
        c.close()
