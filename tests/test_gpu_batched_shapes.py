"""Shapes of the batched solve that follow from the systems' sizes.

The clusters' threads (256, 512, 1024) and the rows below which one CTA solves
a system come from the largest system's share of the rows, and the product
from the longest row.  Each case gives every system the oracle's solution:
x is compared with the host restatement of itl::cg at the same tolerance.  Both
stop at ||r|| <= rtol ||b||, so they differ by at most 2 rtol cond(A): the
graphs' shifted Laplacians (shift 0.01 of the degree) have cond <= 2 deg / (0.01
deg) = 200 after diagonal scaling, and 2e-10 * 200 is 4e-8.
"""
import numpy as np
import pytest

# sizes of the systems; 148 SMs of 1024 threads are divided by share of rows
CASES = {
    "256": [90] * 80 + [130] * 3,             # share ~2,000 threads: small and large
    "512": [300] * 22 + [900, 40, 33, 1],     # ~7,000
    "1024": [700, 257, 3],                    # most of the chip
    "one": [1000],
}


def _batch(M, sizes, dense):
    g = np.random.default_rng(4)
    rps, cis, vs, off = [np.zeros(1, np.int64)], [], [], [0]
    for k, ns in enumerate(sizes):
        if ns < 8:   # too small for a graph: a diagonal
            rp, ci, v = np.arange(ns + 1), np.arange(ns), g.uniform(1.0, 2.0, ns)
        else:
            _, rp, ci, v = M.random_graph(ns, 6.0, 1e-2, k + 1)
        if dense and k == 0:   # a row and column longer than the stream's chunk
            a = np.zeros((ns, ns))
            for i in range(ns):
                a[i, ci[rp[i]:rp[i + 1]]] = v[rp[i]:rp[i + 1]]
            a[0, 1:] = a[1:, 0] = -0.01
            a[np.arange(ns), np.arange(ns)] = 0
            d = np.abs(a).sum(1)
            a[np.arange(ns), np.arange(ns)] = 1.01 * d
            ri, ci = np.nonzero(a)
            rp, v = np.searchsorted(ri, np.arange(ns + 1)), a[ri, ci]
        rps.append(rps[-1][-1] + np.asarray(rp[1:], np.int64))
        cis.append(np.asarray(ci) + off[-1])
        vs.append(v)
        off.append(off[-1] + ns)
    rp = np.concatenate(rps).astype(np.int32)
    return rp, np.concatenate(cis).astype(np.int32), np.concatenate(vs), np.asarray(off, np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("name", list(CASES))
def test_shapes_by_size(M, ctx, restate, name, dense, mode):
    if dense and name == "256":
        pytest.skip("its rows are shorter than the chunk")
    rp, ci, v, off = _batch(M, CASES[name], dense)
    n = len(rp) - 1
    b = M.normal(n, 8)
    A = M.Csr(ctx, rp, ci, v)
    P = M.Pc(A, "diagonal", M.FP32 if mode == "mixed" else M.FP64)
    x, db = ctx.to_device(np.zeros(n)), ctx.to_device(b)
    kw = dict(mode=M.SOLVE_MIXED, inner_rtol=1e-5) if mode == "mixed" else {}
    st, res = M.solve_batched(A, P, off, x, db, rtol=1e-10, max_iter=4000, **kw)
    assert st == M.OK and all(r.kernel_launches == 1 for r in res)
    got = x.download()
    for s in range(len(off) - 1):
        a, e = off[s], off[s + 1]
        sub = (e - a, rp[a:e + 1] - rp[a], ci[rp[a]:rp[e]] - a, v[rp[a]:rp[e]])
        ref = restate.solve("cg", "diagonal", sub, b[a:e], rtol=1e-10, max_iter=4000)
        assert ref["err"] == 0 and res[s].error == 0
        if mode == "fp64":
            assert abs(res[s].iterations - ref["iterations"]) <= 2
        assert np.linalg.norm(got[a:e] - ref["x"]) <= 4e-8 * np.linalg.norm(ref["x"]), s
