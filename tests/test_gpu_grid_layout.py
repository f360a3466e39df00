"""Products, Jacobi-applied factors and solves on the grid layout (at most 32
distinct offsets column - row, values by offset, a mask per row) against the
32-bit index layout (MTLGPU_SELL_INDEX=32) and the oracle: row sums in the
reference's order (mat_vec_mult.hpp:666-688), bit for bit.  Row counts around the
slices and warps, offset counts with kernels of their own and others, up to the
32 that fit and one more, rows lacking offsets, vectors off the 16-byte grid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def offsets_matrix(n, offs, drop, seed):
    """CSR with entries (r, r + o) for o in offs where they exist, each left out
    with probability `drop` (never the diagonal)."""
    g = np.random.default_rng(seed)
    rows, cols = [], []
    for o in sorted(offs):
        r = np.arange(max(0, -o), min(n, n - o))
        if o and drop:
            r = r[g.random(len(r)) >= drop]
        rows.append(r)
        cols.append(r + o)
    r, c = np.concatenate(rows), np.concatenate(cols)
    k = np.lexsort((c, r))
    r, c = r[k], c[k]
    v = g.uniform(-1, 1, len(r))
    v[r == c] = 2.0 * len(offs)
    rp = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(r, minlength=n), out=rp[1:])
    return n, rp, c.astype(np.int32), v


SYM = {3: [1], 5: [1, 40], 7: [1, 40, 300], 9: [1, 39, 40, 41], 11: [1, 2, 5, 40, 77],
       27: [1, 9, 10, 11, 90, 91, 92, 99, 100, 101, 110, 111, 112], 31: list(range(3, 33, 2))}


def sym(w):
    return [0] + SYM[w] + [-o for o in SYM[w]]


CASES = ([(n, sym(7), 0.0) for n in (301, 383, 384, 385, 640, 1000, 4097)] +
         [(2500, sym(w), 0.1) for w in (3, 5, 7, 9, 11, 27, 31)] +
         [(3000, sym(31) + [200], 0.0), (3000, sym(31) + [200, 201], 0.0), (129, [0], 0.0),
          (900, [0, 1, 2, 700], 0.0), (900, [-880, -3, 0], 0.0)])


@pytest.mark.parametrize("n,offs,drop", CASES)
@pytest.mark.parametrize("shift", [0, 1])
def test_products_bit_exact(M, ctx, restate, n, offs, drop, shift):
    A = offsets_matrix(n, offs, drop, n)
    dA = M.Csr(ctx, *A[1:])
    x = M.uniform(n, 3)
    x[n // 2] = np.inf          # rows without an entry there must not see it
    big, y = ctx.array(n + shift), ctx.array(n + shift)
    big.upload(np.concatenate([np.zeros(shift), x]))

    class View:                 # a vector `shift` elements into an allocation
        def __init__(self, a):
            self.n, self.ptr = n, M.C.c_void_p(a.ptr.value + 8 * shift)
    dA.spmv(View(big), View(y))
    assert np.array_equal(y.download()[shift:], restate.spmv(A, x), equal_nan=True)
    dA.spmv(View(big), View(y), 2.0, -0.5)
    with np.errstate(invalid="ignore"):
        want = -0.5 * restate.spmv(A, x) + 2.0 * restate.spmv(A, x)
    assert np.allclose(y.download()[shift:], want, rtol=1e-15, atol=1e-13, equal_nan=True)
    dA.close()


@pytest.mark.parametrize("n,offs,drop", CASES)
def test_same_as_indexed_layout(M, monkeypatch, n, offs, drop):
    A = offsets_matrix(n, sorted(set(offs) | {-o for o in offs}), 0.0, n + 1)
    sym_v = {}
    for r in range(n):
        for j in range(A[1][r], A[1][r + 1]):
            key = (min(r, A[2][j]), max(r, A[2][j]))
            A[3][j] = sym_v.setdefault(key, A[3][j])
    out = {}
    for layout in ("grid", "32"):
        if layout == "32":
            monkeypatch.setenv("MTLGPU_SELL_INDEX", "32")
        c = M.Context(0)
        dA = M.Csr(c, *A[1:])
        P = M.Pc(dA, "ic0", M.FP32)
        P.set_jacobi_sweeps(2)
        r64, r32 = M.uniform(n, 5), M.uniform(n, 6).astype(np.float32)
        a, z = c.to_device(r64), c.array(n)
        P.apply(a, z)
        a32, z32 = c.to_device(r32), c.array(n, np.float32)
        P.apply_f32(a32, z32)
        y32 = c.array(n, np.float32)
        dA.spmv_f32(a32, y32)
        b, x = c.to_device(r64), c.to_device(np.zeros(n))
        st, res, _ = M.solve("cg", dA, P, x, b, rtol=1e-10, max_iter=500, mode=M.SOLVE_MIXED)
        assert st == M.OK
        Q = M.Pc(dA, "ilu0")
        Q.set_jacobi_sweeps(1)
        x2 = c.to_device(np.zeros(n))
        st, res2, _ = M.solve("bicgstab", dA, Q, x2, b, rtol=1e-10, max_iter=500)
        assert st == M.OK
        out[layout] = [v.download() for v in (z, z32, y32, x, x2)]
        P.close(), Q.close(), dA.close(), c.close()
    for k in range(3):          # one fixed order of operations per row
        assert np.array_equal(out["grid"][k], out["32"][k]), k
    for k in (3, 4):            # dot products are grouped differently
        ref = np.linalg.norm(out["32"][k])
        assert np.linalg.norm(out["grid"][k] - out["32"][k]) <= 1e-8 * ref
