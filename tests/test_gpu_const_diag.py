"""GPU: matrices whose diagonals hold one value each (constant-coefficient
stencils), whose FP64 SpMV reads no values, against the CSR kernel.

Rows are summed in the same order with the same products either way, so every
comparison is of bits; an infinite entry of x reaches only the rows that have
an entry in its column.
"""
import numpy as np
import pytest

from solver_cpp_b200.matrices import CSR, convdiff3d, poisson2d, poisson3d

pytestmark = pytest.mark.gpu


def bands(n, coefs):
    """Every row's entries at the offsets of `coefs` that exist."""
    offs = sorted(coefs)
    i = np.arange(n)
    has = np.stack([(i + o >= 0) & (i + o < n) for o in offs], 1)
    ptr = np.zeros(n + 1, dtype=np.int32)
    ptr[1:] = np.cumsum(has.sum(1))
    return CSR(ptr, (i[:, None] + np.array(offs))[has].astype(np.int32),
               np.broadcast_to([coefs[o] for o in offs], has.shape)[has].copy())


CASES = {
    "poisson2d_61": lambda: poisson2d(61),
    "poisson3d_37x20x9": lambda: poisson3d(37, 20, 9),
    "convdiff3d_33": lambda: convdiff3d(33),
    "tridiagonal": lambda: bands(1000, {-1: -1.0, 0: 2.5, 1: -1.25}),
    "eight": lambda: bands(777, {-40: 0.3, -9: -1.0, -2: 0.0, 0: 4.0, 1: -0.5, 3: 1e-300, 40: 1.0, 41: -2.0}),
    "one_row": lambda: bands(1, {0: 3.0}),
}


@pytest.mark.parametrize("changed", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_spmv_bits(ks, ctx, name, changed):
    A = CASES[name]()
    if changed and A.nnz > 1:  # one entry differs: the values are read again
        A.val[A.nnz // 2] = np.nextafter(A.val[A.nnz // 2], 9.0)
    x = np.random.default_rng(1).standard_normal(A.n)
    x[A.n // 3] = np.inf
    D, C = ctx.matrix(A, transpose=True), ctx.matrix(A, transpose=True, diag=False)
    assert D.info()["diagonals"] > 0 and C.info()["diagonals"] == 0
    X, Y = ctx.vector(x), ctx.vector(n=A.n)
    for trans in (False, True):
        ks.spmv(D, X, Y, trans=trans)
        got = Y.numpy()
        ks.spmv(C, X, Y, trans=trans)
        assert np.array_equal(got.view(np.int64), Y.numpy().view(np.int64)), trans


@pytest.mark.parametrize("method,prob,L", [("CG", (100, 100, 90), 30), ("CR", (37, 41, 43), 30), ("BICG", 41, 30)])
def test_on_chip_solves(ks, ctx, method, prob, L):
    """The on-chip kernels with the diagonals' values as parameters and as
    arrays (one entry one ulp off, which moves the solution by rounding only)."""
    A = convdiff3d(prob) if isinstance(prob, int) else poisson3d(*prob)
    b = np.random.default_rng(2).standard_normal(A.n)
    xs = []
    for changed in (False, True):
        if changed:
            A.val[A.nnz // 2] = np.nextafter(A.val[A.nnz // 2], 9.0)
        M = ctx.matrix(A, transpose=True)
        r = ks.solve(ctx, M, method, b, E=1e-14, L=L, cluster_solve=0, profile=1)
        assert r.report["n_mv"] == 1, r.report
        xs.append(r)
        M.close()
    assert np.allclose(xs[0].hist_err, xs[1].hist_err, rtol=1e-9, atol=0)
    assert np.linalg.norm(xs[0].x - xs[1].x) <= 1e-9 * np.linalg.norm(xs[1].x)
