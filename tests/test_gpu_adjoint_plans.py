"""The transposed ILU(0) factors of a stencil matrix: U^T is swept along grid
lines and keeps no level-ordered plan beside its records, so the first adjoint
apply takes no more device memory than with level-ordered sweeps alone
(MTLGPU_SWEEP=ticket), and gives the same bits."""
import numpy as np
import pytest

from test_gpu_line_sweep import context

pytestmark = pytest.mark.gpu


def test_adjoint_plans_are_made_once(M):
    import torch
    n, rp, ci, v = M.convdiff27(96, 2)
    r = M.uniform(n, 3)
    took, got = {}, {}
    for mode in (None, "ticket"):
        c = context(M, mode)
        try:
            A = M.Csr(c, rp, ci, v)
            P = M.Pc(A, "ilu0", M.FP32)
            x, y = c.to_device(r), c.array(n)
            P.apply(x, y)       # the other plans are there
            before = torch.cuda.mem_get_info(0)[0]
            P.adjoint_apply(x, y)
            took[mode] = before - torch.cuda.mem_get_info(0)[0]
            got[mode] = y.download()
            P.close(), A.close()
        finally:
            c.close()
    assert np.array_equal(got[None], got["ticket"])
    assert took[None] <= took["ticket"], took
