"""GPU: CG of matrices without a diagonal copy as one on-chip launch
(ks_csr_cg.cuh), against the kernel-per-step engine.

The product adds every row's entries in the CSR kernel's order, and the vector
updates are the engine's; only the dot products add their terms in another
order. On these systems (diagonally dominant by 5 %) the first 40 iterations of
the two paths therefore agree to 1e-9, as in test_gpu_chip_cg.py.
"""
import numpy as np
import pytest

from solver_cpp_b200.matrices import CSR

pytestmark = pytest.mark.gpu


def graph(n, lower, upper, deg, seed=0, empty=(), skew=0.0):
    """Random entries between `lower` rows before and `upper` rows after the
    row (symmetric for lower == upper), rows of up to `deg` pairs; rows in
    `empty` keep their diagonal only."""
    rng = np.random.default_rng(seed)
    m = rng.integers(0, deg + 1, n)
    i = np.repeat(np.arange(n), m)
    j = i + 1 + rng.integers(0, max(min(lower, upper), 1), i.size)
    keep = (j < n) & ~np.isin(i, empty) & ~np.isin(j, empty)
    key = np.unique(i[keep] * n + j[keep])
    i, j = key // n, key % n
    w = -rng.uniform(0.5, 1.0, i.size)
    ri, ci, vi = [i, j], [j, i], [w, w + skew]
    if upper > lower:  # the far ends of the offsets, one entry each way where allowed
        ri.append(np.array([0])), ci.append(np.array([upper])), vi.append(np.array([-0.25]))
    rows, cols, vals = np.concatenate(ri), np.concatenate(ci), np.concatenate(vi)
    d = 1.05 * np.bincount(rows, weights=-vals, minlength=n) + 0.1
    rows, cols, vals = np.concatenate([rows, np.arange(n)]), np.concatenate([cols, np.arange(n)]), np.concatenate([vals, d])
    order = np.argsort(rows * n + cols, kind="stable")
    ptr = np.zeros(n + 1, dtype=np.int32)
    ptr[1:] = np.cumsum(np.bincount(rows, minlength=n))
    return CSR(ptr, cols[order].astype(np.int32), vals[order])


def both(ks, ctx, A, L=40, **kw):
    M = ctx.matrix(A, **kw)
    assert M.info()["diagonals"] == 0
    b = np.random.default_rng(1).standard_normal(A.n)
    chip = ks.solve(ctx, M, "CG", b, E=1e-14, L=L, cluster_solve=0, profile=1)
    step = ks.solve(ctx, M, "CG", b, E=1e-14, L=L, cluster_solve=1)
    M.close()
    return chip, step


def agree(chip, step):
    assert chip.status == step.status and chip.loop == step.loop, (chip.status, step.status, chip.loop, step.loop)
    assert np.allclose(chip.hist_err, step.hist_err, rtol=1e-9, atol=0)
    assert np.linalg.norm(chip.x - step.x) <= 1e-9 * np.linalg.norm(step.x)


# 8,193 rows: the smallest of this path; 16,384 / 16,385 and 65,536 / 65,537
# rows: the launch shape changes; 606,208 = 148 x 4,096: the largest; degrees
# down to rows without neighbours, windows from a few rows to the largest
@pytest.mark.parametrize("n,band,deg", [(8193, 3, 2), (8200, 8000, 7), (16384, 500, 7), (16385, 1, 1), (65536, 9000, 4),
                                        (65537, 700, 10), (250007, 6000, 6), (606208, 2000, 2)])
def test_against_engine(ks, ctx, n, band, deg):
    chip, step = both(ks, ctx, graph(n, band, band, deg, empty=(0, 31, 32, n // 2, n - 1)))
    assert chip.report["n_mv"] == 1 and chip.report["n_dot"] == 0, chip.report
    agree(chip, step)


def test_unequal_window_and_unsymmetric_values(ks, ctx):
    chip, step = both(ks, ctx, graph(30011, 900, 5000, 5, skew=0.02), L=15)
    assert chip.report["n_mv"] == 1
    agree(chip, step)


@pytest.mark.parametrize("L", [0, 1])
def test_stops_at_maxloop(ks, ctx, L):
    agree(*both(ks, ctx, graph(9001, 300, 300, 5), L=L))


def test_what_does_not_fit_takes_the_engine(ks, ctx):
    """A window wider than shared memory, int32 columns, one very long row
    (slices more than twice the nonzeros): no slices or no launch, same solve."""
    for A, kw in ((graph(70000, 30000, 30000, 4), {}), (graph(20000, 300, 300, 4), dict(index32=True))):
        chip, step = both(ks, ctx, A, L=10, **kw)
        assert chip.report["n_mv"] != 1  # many products, or none by that name in one cluster
        agree(chip, step)
    n = 40000
    A = graph(n, 10, 10, 1)
    long = CSR(np.concatenate([[0], A.ptr[1:] + 9000]).astype(np.int32),
               np.concatenate([np.arange(9000 + A.ptr[1]), A.col[A.ptr[1]:]]).astype(np.int32),
               np.concatenate([np.full(9000 + A.ptr[1], -1e-6), A.val[A.ptr[1]:]]))
    long.val[0] = 2.0
    chip, step = both(ks, ctx, long, L=10)
    agree(chip, step)


def test_converges_to_the_solution(ks, ctx, oracle):
    A = graph(9500, 400, 400, 6)
    b = np.random.default_rng(4).standard_normal(A.n)
    M = ctx.matrix(A)
    r = ks.solve(ctx, M, "CG", b, E=1e-12)
    o = oracle.solve(A, b, "CG", E=1e-12)
    assert r.converged and o["status"] == 0 and abs(r.loop - o["loop"]) <= 1
    # both residuals are 1e-12 |b|, the smallest eigenvalue is 0.1 at least
    assert np.linalg.norm(r.x - o["x"]) <= 2.5e-11 * np.linalg.norm(b)
    M.close()
