"""Workloads of the sparse iterative-solve path, for timing and comparison.

Each case is the work of one user call (or of the short sequence a user's
program makes of it) through the Python binding of the C ABI: residuals and
products, triangular applies, Krylov solves in FP64 and in mixed precision, a
batch of independent systems, a differentiable solve with its gradients, and
the way from element contributions to a solution.  Vectors are torch tensors
on the GPU, as a PyTorch program has them; the context works on a torch
stream.

Right-hand sides are made from a known solution (b = A x_true, formed by plain
torch / numpy or by the host generators), so a solve's exact answer is x_true.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "mtl4-mirror_b200", "python"))
import mtlgpu as M  # noqa: E402

INNER_RTOL = 1e-5   # FP32 inner solves of the mixed mode, as the benchmark asks


# ---- cases ------------------------------------------------------------------
def listed():
    return [
        # the smallest calls: residual and its norm on the 100 x 100 Laplacian
        # (the grid of the reference's ic_0_cg example): launch latency
        dict(name="residual_lap2d_100x100", kind="residual", m=100, n=100),
        # y = A x on the large stencil matrix of the headline solve
        dict(name="spmv_lap3d_128", kind="spmv", grid="lap3d", N=128, prec="fp64"),
        # y = A x on an irregular matrix (random graph Laplacian pattern)
        dict(name="spmv_graph_200k", kind="spmv", grid="graph", N=200003, deg=14, prec="fp64"),
        # z = solve(P, r): exact IC(0) triangular solves, as one user call
        dict(name="apply_ic0_lap3d_96", kind="apply", grid="lap3d", N=96),
        # the reference's own example: PCG-IC(0), FP64, exact sweeps
        dict(name="cg_ic0_lap2d_100x100", kind="solve", method="cg", pc="ic0", grid="lap2d",
             m=100, n=100, mode="fp64", jacobi=0),
        # the same at full size: the reference's arithmetic on 128^3
        dict(name="cg_ic0_lap3d_128", kind="solve", method="cg", pc="ic0", grid="lap3d", N=128,
             mode="fp64", jacobi=0),
        # the benchmark's headline solve: FP32 inner, Jacobi-applied IC(0)
        dict(name="cg_mixed_lap3d_128", kind="solve", method="cg", pc="ic0", grid="lap3d", N=128,
             mode="mixed", jacobi=1),
        # unsymmetric 27-point convection-diffusion, mixed precision
        dict(name="bicgstab_mixed_cd27_96", kind="solve", method="bicgstab", pc="ilu0",
             grid="cd27", N=96, mode="mixed", jacobi=1),
        # another Krylov method with exact ILU(0) solves, an odd grid
        dict(name="tfqmr_ilu0_cd27_47", kind="krylov", method="tfqmr", param=0, N=47),
        # independent random-graph systems in one batched call
        dict(name="batched_diag_96", kind="batched", count=96, pc="diagonal"),
        # differentiable finite-volume solve: forward, adjoint, value gradients
        dict(name="adjoint_fv2d_512", kind="adjoint", N=512, jacobi=2),
        # element contributions -> matrix -> IC(0) -> mixed solve
        dict(name="assemble_solve_64", kind="assemble", N=64),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["residual", "spmv", "apply", "solve", "solve", "mixed", "mixed", "krylov",
                       "batched", "adjoint", "assemble"])
    if kind == "residual":
        return dict(kind=kind, m=_log(rng, 30, 500), n=_log(rng, 30, 500))
    if kind == "spmv":
        grid = rng.choice(["lap2d", "lap3d", "cd27", "fv2d", "graph"])
        prec = rng.choice(["fp64", "fp64", "fp32"])
        if grid == "lap2d":
            return dict(kind=kind, grid=grid, m=_log(rng, 100, 1500), n=_log(rng, 100, 1500),
                        prec=prec)
        if grid == "graph":
            return dict(kind=kind, grid=grid, N=_log(rng, 20000, 300000), deg=rng.randint(6, 24),
                        prec=prec)
        N = {"lap3d": (24, 128), "cd27": (16, 80), "fv2d": (100, 1200)}[grid]
        return dict(kind=kind, grid=grid, N=_log(rng, *N), prec=prec)
    if kind == "apply":
        if rng.random() < 0.5:
            return dict(kind=kind, grid="lap3d", N=_log(rng, 16, 110))
        return dict(kind=kind, grid="lap2d", m=_log(rng, 40, 700), n=_log(rng, 40, 700))
    if kind == "solve":
        grid = rng.choice(["lap2d", "lap3d", "cd27"])
        if grid == "lap2d":
            return dict(kind=kind, method="cg", pc=rng.choice(["ic0", "ic0", "diagonal"]),
                        grid=grid, m=_log(rng, 30, 220), n=_log(rng, 30, 220), mode="fp64",
                        jacobi=0)
        if grid == "lap3d":
            return dict(kind=kind, method="cg", pc=rng.choice(["ic0", "ic0", "diagonal", "none"]),
                        grid=grid, N=_log(rng, 12, 100), mode="fp64", jacobi=0)
        return dict(kind=kind, method="bicgstab", pc="ilu0", grid=grid, N=_log(rng, 12, 60),
                    mode="fp64", jacobi=0)
    if kind == "mixed":
        if rng.random() < 0.6:
            return dict(kind="solve", method="cg", pc="ic0", grid="lap3d", N=_log(rng, 20, 127),
                        mode="mixed", jacobi=rng.choice([1, 1, 2]))
        return dict(kind="solve", method="bicgstab", pc="ilu0", grid="cd27", N=_log(rng, 14, 90),
                    mode="mixed", jacobi=rng.choice([1, 1, 2]))
    if kind == "krylov":
        method, param = rng.choice([("cgs", 0), ("bicgstab_2", 0), ("bicgstab_ell", 4),
                                    ("tfqmr", 0)])
        return dict(kind=kind, method=method, param=param, N=_log(rng, 12, 50))
    if kind == "batched":
        return dict(kind=kind, count=rng.randint(16, 90), pc=rng.choice(["diagonal", "none"]))
    if kind == "adjoint":
        if rng.random() < 0.6:
            return dict(kind=kind, N=_log(rng, 64, 500), jacobi=2)
        return dict(kind=kind, N=_log(rng, 40, 110), jacobi=0)
    return dict(kind=kind, N=_log(rng, 12, 80))


# ---- inputs -----------------------------------------------------------------
class _Vec(M.DeviceArray):
    """A torch tensor as the binding's device array (the memory is torch's)."""

    def __init__(self, ctx, t):
        self.ctx, self.t, self.n = ctx, t, t.numel()
        self.dtype = np.dtype(str(t.dtype).replace("torch.", ""))
        self.ptr = M.C.c_void_p(t.data_ptr())

    def free(self):
        self.ptr = M.C.c_void_p()


def _vec(ctx, a):
    return _Vec(ctx, torch.as_tensor(a, device="cuda"))


def _new(ctx, n, dtype=torch.float64):
    return _Vec(ctx, torch.zeros(n, dtype=dtype, device="cuda"))


def _uniform(seed, n, tag=0):
    return np.random.default_rng([int(seed), tag]).uniform(-1.0, 1.0, n)


def _dims(c):
    return (c["m"], c["n"]) if "m" in c else (c["N"],) * 3


def _lap_mult(dims, x):
    """A x of the 5- / 7-point Laplacian on a grid in natural order."""
    x = x.reshape(dims)
    y = 2.0 * len(dims) * x
    for d in range(len(dims)):
        lo = [slice(None)] * len(dims)
        hi = list(lo)
        lo[d], hi[d] = slice(0, -1), slice(1, None)
        y[tuple(lo)] -= x[tuple(hi)]
        y[tuple(hi)] -= x[tuple(lo)]
    return y.reshape(-1)


def _graphs(ns, degs, seed):
    """Block-diagonal CSR of symmetric random graphs' shifted Laplacians: graph
    k has ns[k] vertices and average degree about degs[k] (rows sorted)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    ns = torch.as_tensor(ns, dtype=torch.int64, device="cuda")
    degs = torch.as_tensor(degs, dtype=torch.float64, device="cuda")
    off = torch.cumsum(ns, 0) - ns
    n = int(ns.sum())
    edges = (ns * degs / 2).to(torch.int64)
    size, base = (torch.repeat_interleave(t, edges) for t in (ns, off))
    r, q = (base + torch.minimum((torch.rand(len(size), generator=g, device="cuda",
                                             dtype=torch.float64) * size).to(torch.int64),
                                 size - 1) for _ in range(2))
    keep = r != q
    r, q = r[keep], q[keep]
    d = torch.arange(n, device="cuda", dtype=torch.int64) * (n + 1)
    key = torch.unique(torch.cat([r * n + q, q * n + r, d]))
    r, q = key // n, key % n
    cnt = torch.bincount(r, minlength=n)
    v = torch.where(r == q, (cnt - 1 + 0.01 * torch.repeat_interleave(degs, ns))[r].to(
        torch.float64), torch.tensor(-1.0, dtype=torch.float64, device="cuda"))
    rp = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), torch.cumsum(cnt, 0)])
    return rp.to(torch.int32).cpu().numpy(), q.to(torch.int32).cpu().numpy(), v.cpu().numpy()


def _batch(c):
    """Sizes (spread log-uniformly, mixed order) and degrees of the batch's
    systems; the graphs themselves come from the seed."""
    g = np.random.default_rng(5)
    t = (np.arange(c["count"]) + 0.5) / c["count"]
    ns = np.exp(math.log(1000) + t * math.log(65536 / 1000)).astype(np.int64)
    return g.permutation(ns), g.uniform(8.0, 32.0, c["count"])


def _host_matrix(c, seed):
    """(rp, ci, v) of the generated matrices; None for the Laplacians."""
    if c["grid"] == "cd27":
        return M.convdiff27(c["N"], seed)[1:]
    if c["grid"] == "fv2d":
        return M.fv2d(c["N"], seed=seed)[1:]
    if c["grid"] == "graph":
        return _graphs([c["N"]], [float(c["deg"])], seed)
    return None


def _matrix(ctx, c, seed):
    h = _host_matrix(c, seed)
    if h is not None:
        return M.Csr(ctx, *h), h
    if c["grid"] == "lap2d":
        return M.Csr.laplacian2d(ctx, c["m"], c["n"]), None
    return M.Csr.laplacian3d(ctx, c["N"]), None


def _mult(c, h, x):
    return _lap_mult(_dims(c), x) if h is None else M.csr_mult((len(h[0]) - 1,) + tuple(h), x)


def _rows(c):
    if c["kind"] == "assemble":
        return c["N"] ** 3
    if c["kind"] == "adjoint" or c.get("grid") == "fv2d":
        return c["N"] ** 2
    if c.get("grid") == "graph":
        return c["N"]
    return int(np.prod(_dims(c)))


def _links(N, seed):
    """Link conductances of an N^3 grid: weights of the edges of each direction."""
    g = np.random.default_rng([int(seed), 11])
    return [g.uniform(0.5, 1.5, tuple(N - (d == a) for a in range(3))) for d in range(3)]


def _pair(d):
    lo, hi = [slice(None)] * 3, [slice(None)] * 3
    lo[d], hi[d] = slice(0, -1), slice(1, None)
    return tuple(lo), tuple(hi)


def prepare(case, seed):
    c = dict(case)
    stream = torch.cuda.Stream()
    ctx = M.Context(0, stream.cuda_stream)
    s = dict(c=c, ctx=ctx, stream=stream)
    k = c["kind"]
    if k == "batched":
        ns, degs = _batch(c)
        rp, ci, v = _graphs(ns, degs, seed)
        n = len(rp) - 1
        s["A"], s["off"] = M.Csr(ctx, rp, ci, v), np.concatenate([[0], np.cumsum(ns)])
        s["b"] = _vec(ctx, M.csr_mult((n, rp, ci, v), _uniform(seed, n)))
        s["x"] = _new(ctx, n)
        s["P"] = None if c["pc"] == "none" else M.Pc(s["A"], c["pc"])
    elif k == "assemble":
        N = c["N"]
        idx = np.arange(N ** 3, dtype=np.int32).reshape(N, N, N)
        x = _uniform(seed, N ** 3).reshape(N, N, N)
        r, q, v = [idx.ravel()], [idx.ravel()], [np.full(N ** 3, 0.05)]
        y = 0.05 * x
        for d, w in enumerate(_links(N, seed)):  # 2 x 2 element contributions per link
            lo, hi = _pair(d)
            a, b, w1 = idx[lo].ravel(), idx[hi].ravel(), w.ravel()
            r += [a, a, b, b]
            q += [a, b, a, b]
            v += [w1, -w1, -w1, w1]
            f = w * (x[lo] - x[hi])
            y[lo] += f
            y[hi] -= f
        s["trip"] = [_vec(ctx, np.concatenate(t)) for t in (r, q, v)]
        s["b"], s["x"] = _vec(ctx, y.ravel()), _new(ctx, N ** 3)
    elif k == "adjoint":
        c["grid"] = "fv2d"
        s["A"], h = _matrix(ctx, c, seed)
        n = len(h[0]) - 1
        s["P"] = M.Pc(s["A"], "ic0")
        if c["jacobi"]:
            s["P"].set_jacobi_sweeps(c["jacobi"])
        s["b"] = _vec(ctx, _mult(c, h, _uniform(seed, n)))
        s["g"] = _vec(ctx, _mult(c, h, _uniform(seed, n, 1)))   # A is symmetric
        s["x"], s["lam"], s["grad"] = _new(ctx, n), _new(ctx, n), _new(ctx, len(h[1]))
    else:
        c.setdefault("grid", "lap2d" if k == "residual" else "cd27")
        s["A"], h = _matrix(ctx, c, seed)
        n = s["A"].n
        xt = _uniform(seed, n)
        if k == "residual":
            s["x"], s["b"] = _vec(ctx, xt), _vec(ctx, _uniform(seed, n, 1))
            s["r"] = _new(ctx, n)
        elif k == "spmv":
            dt = torch.float32 if c["prec"] == "fp32" else torch.float64
            s["x"] = _vec(ctx, torch.as_tensor(xt).to(dt))
            s["y"] = _new(ctx, n, dt)
            if c["prec"] == "fp32":
                s["A"].spmv_f32(s["x"], s["y"])   # the float copy of A's values is kept
        elif k == "apply":
            s["P"] = M.Pc(s["A"], "ic0")
            s["b"], s["x"] = _vec(ctx, xt), _new(ctx, n)
        else:
            s["P"] = None
            if k == "krylov":
                s["P"] = M.Pc(s["A"], "ilu0")
            elif c["pc"] != "none":
                s["P"] = M.Pc(s["A"], c["pc"], M.FP32 if c["mode"] == "mixed" else M.FP64)
                if c["jacobi"]:
                    s["P"].set_jacobi_sweeps(c["jacobi"])
            s["b"], s["x"] = _vec(ctx, _mult(c, h, xt)), _new(ctx, n)
    torch.cuda.synchronize()
    return s


# ---- one pass ---------------------------------------------------------------
def _mixed(mode):
    return dict(mode=M.SOLVE_MIXED, inner_rtol=INNER_RTOL) if mode == "mixed" else {}


def _zero(s, *names):
    """The initial guess, on the context's stream."""
    with torch.cuda.stream(s["stream"]):
        for n in names:
            s[n].t.zero_()


def _ok(status):
    if status != M.OK:
        raise RuntimeError("solve: status %d" % status)


def run(s):
    c, ctx = s["c"], s["ctx"]
    k = c["kind"]
    if k == "residual":     # r = b - A x and its norm (read by the host)
        s["A"].spmv(s["x"], s["r"], -1.0, 0.0)
        ctx.axpy(1.0, s["b"], s["r"])
        return {"r": s["r"].t, "norm": ctx.two_norm(s["r"])}
    if k == "spmv":
        if c["prec"] == "fp32":
            s["A"].spmv_f32(s["x"], s["y"])
        else:
            s["A"].spmv(s["x"], s["y"])
        return {"y": s["y"].t}
    if k == "apply":
        s["P"].apply(s["b"], s["x"])
        return {"z": s["x"].t}
    if k == "solve":
        _zero(s, "x")
        _ok(M.solve(c["method"], s["A"], s["P"], s["x"], s["b"], rtol=1e-10, max_iter=4000,
                    **_mixed(c["mode"]))[0])
        return {"x": s["x"].t}
    if k == "krylov":
        _zero(s, "x")
        _ok(M.solve_krylov(c["method"], s["A"], s["P"], s["x"], s["b"], param=c["param"],
                           rtol=1e-10, max_iter=2000)[0])
        return {"x": s["x"].t}
    if k == "batched":
        _zero(s, "x")
        _ok(M.solve_batched(s["A"], s["P"], s["off"], s["x"], s["b"], rtol=1e-8,
                            max_iter=5000)[0])
        return {"x": s["x"].t}
    if k == "adjoint":
        _zero(s, "x", "lam")
        for x, b in (("x", "b"), ("lam", "g")):
            _ok(M.solve("cg", s["A"], s["P"], s[x], s[b], rtol=1e-12, max_iter=20000)[0])
        s["A"].values_grad(s["lam"], s["x"], s["grad"])
        return {"x": s["x"].t, "lambda": s["lam"].t, "grad": s["grad"].t}
    n = s["x"].n            # assemble: a new matrix from its element contributions
    _zero(s, "x")
    A = M.Csr.assemble(ctx, n, n, *s["trip"], updater=M.UPDATE_PLUS)
    P = M.Pc(A, "ic0", M.FP32)
    P.set_jacobi_sweeps(1)
    st = M.solve("cg", A, P, s["x"], s["b"], rtol=1e-10, max_iter=4000, **_mixed("mixed"))[0]
    P.close()
    A.close()
    _ok(st)
    return {"x": s["x"].t}


# ---- what a pass cannot do without ------------------------------------------
def work(case):
    """Bytes: vectors and the matrix read once, results written once; for a
    solve, the matrix, the factors and the vectors of every iteration it is
    known to need (a bound from the problem's size, not the present count)."""
    c = dict(case)
    k = c["kind"]
    if k == "batched":
        n, nnz = 15400 * c["count"], 15400 * 21 * c["count"]
        its, tri, v = 17, 0, 8
    else:
        n = _rows(c)
        g = {"krylov": "cd27", "adjoint": "fv2d", "assemble": "lap3d",
             "residual": "lap2d"}.get(k, c.get("grid"))
        nnz = n * {"lap2d": 5, "fv2d": 5, "lap3d": 7, "cd27": 27, "graph": c.get("deg", 0) + 1}[g]
        tri = nnz - n
        v = 4 if c.get("mode") == "mixed" or k == "assemble" or c.get("prec") == "fp32" else 8
        side = n ** (1 / 3) if g in ("lap3d", "cd27") else n ** 0.5
        its = max(4.0, {"lap2d": 0.95, "fv2d": 1.6, "lap3d": 1.0, "cd27": 0.45,
                        "graph": 0.0}[g] * side)
    mat = nnz * (v + 4) + 4 * n
    if k == "residual":
        return {"bytes": mat + 3 * 8 * n, "flops": 2 * nnz + 4 * n}
    if k == "spmv":
        return {"bytes": mat + 2 * v * n, "flops": 2 * nnz}
    if k == "apply":
        return {"bytes": tri * 12 + 4 * 8 * n, "flops": 2 * tri}
    if c.get("pc") in ("diagonal", "none"):
        tri = 0
    per = mat + tri * (v + 4) + 9 * v * n
    fl = 2 * (nnz + tri) + 12 * n
    if k == "krylov" or c.get("method") == "bicgstab":
        per, fl = 2 * per, 2 * fl
    if k == "adjoint":
        its *= 2
    if k == "assemble":
        return {"bytes": its * per + 13 * n * 16 + 4 * mat, "flops": its * fl}
    return {"bytes": its * per, "flops": its * fl}


# ---- exact results ----------------------------------------------------------
def _ic0_apply(dims, r):
    """(L L^T)^-1 r for the Laplacian's IC(0) as the reference factorises it,
    front by front over the grid (numpy, 64 bits): inv_k = 1 / sqrt(a_kk -
    sum (a_mk inv_m)^2), L = off-diagonals a_mk inv_m, diagonal 1 / inv_k."""
    d = tuple(dims)
    pad = tuple(x + 2 for x in d)
    stride = [int(np.prod(pad[a + 1:])) for a in range(len(d))]
    ix = np.indices(d).reshape(len(d), -1)
    at = sum((ix[a] + 1) * stride[a] for a in range(len(d)))
    level = ix.sum(0)
    order = np.argsort(level, kind="stable")
    cuts = np.flatnonzero(np.diff(level[order])) + 1
    fronts = np.split(at[order], cuts)
    inv, y, z = (np.zeros(int(np.prod(pad))) for _ in range(3))
    y[at] = r
    diag = 2.0 * len(d)
    for f in fronts:
        inv[f] = 1.0 / np.sqrt(diag - sum(inv[f - t] ** 2 for t in stride))
        y[f] = (y[f] + sum(inv[f - t] * y[f - t] for t in stride)) * inv[f]
    for f in reversed(fronts):
        z[f] = (y[f] + inv[f] * sum(z[f + t] for t in stride)) * inv[f]
    return z[at]


def exact(case, seed):
    c = dict(case)
    k = c["kind"]
    if k == "batched":
        return {"x": _uniform(seed, int(_batch(c)[0].sum()))}
    n = _rows(c)
    xt = _uniform(seed, n)
    if k == "residual":
        r = _uniform(seed, n, 1) - _lap_mult(_dims(c), xt)
        return {"r": r, "norm": float(np.linalg.norm(r))}
    if k == "spmv":
        h = _host_matrix(c, seed)
        if c["prec"] == "fp32":
            xt = xt.astype(np.float32).astype(np.float64)
        if h is None:
            return {"y": _lap_mult(_dims(c), xt)}
        rp, ci, v = h
        if c["prec"] == "fp32":
            v = v.astype(np.float32).astype(np.float64)
        return {"y": np.add.reduceat(v * xt[ci], rp[:-1])}
    if k == "apply":
        return {"z": _ic0_apply(_dims(c), xt)}
    if k == "adjoint":
        N, lam = c["N"], _uniform(seed, n, 1)
        i, j = np.divmod(np.arange(n), N)
        col = np.stack([np.where(i > 0, -N, n), np.where(j > 0, -1, n), np.zeros(n, np.int64),
                        np.where(j < N - 1, 1, n), np.where(i < N - 1, N, n)], 1)
        here = col < n
        row = np.broadcast_to(np.arange(n)[:, None], col.shape)
        grad = -lam[row[here]] * xt[(row + col)[here]]
        return {"x": xt, "lambda": lam, "grad": grad}
    return {"x": xt}        # b was made from it

