"""GPU: how the one-launch CG kernels stop other than by converging, each kernel
by name, without faulting the GPU.

* Bounded waits: with a limit of 1 ns (ks_ctx_set_wait_limit) they run out, the
  solve reports KS_TIMEOUT and the context keeps working.
* Breakdown: a skew-symmetric matrix of entries -1, 0, 1 and b = 1. Then
  (p, A p) sums whole numbers of both signs to 0, exactly in any order.
* b = 0: the stopping test is 0 / 0.
"""
import numpy as np
import pytest

from solver_cpp_b200.matrices import CSR
from test_gpu_chip_cg import banded, box
from test_gpu_csr_cg import graph
from test_gpu_tile_cg import constant_box

pytestmark = pytest.mark.gpu

SYSTEMS = {
    "k_cg_chip_one_row": ("k_cg_chip", lambda: box(101, 97)),     # r behind flags
    "k_cg_chip_box": ("k_cg_chip", lambda: box(64, 64, 64)),      # r with tags, tiles
    "k_cg_chip_runs": ("k_cg_chip", lambda: box(700, 701)),       # r with tags, runs of rows
    "k_cg_tile": ("k_cg_tile", lambda: constant_box((93, 91, 90))),
    "k_cg_onchip": ("k_cg_onchip", lambda: box(93, 91, 90)),
    "k_cg_onchip_constant": ("k_cg_onchip", lambda: constant_box((300, 60, 61))),
    "k_cg_csr": ("k_cg_csr", lambda: graph(30011, 900, 900, 5)),
    "k_cg_csr_large": ("k_cg_csr", lambda: graph(400000, 2000, 2000, 2)),
}


@pytest.mark.parametrize("name", sorted(SYSTEMS))
def test_wait_runs_out_and_context_survives(ks, ctx, name):
    kernel, make = SYSTEMS[name]
    A = make()
    M = ctx.matrix(A)
    b = np.random.default_rng(2).standard_normal(A.n)
    ctx.set_wait_limit(1)
    try:
        with pytest.raises(ks.KrylovError) as e:
            ks.solve(ctx, M, "CG", b, E=1e-10, L=5)
        assert e.value.status == 7  # KS_TIMEOUT
        assert ctx.solve_kernel() == kernel
    finally:
        ctx.set_wait_limit(0)
    ctx.synchronize()  # the flag was reported once and cleared
    r = ks.solve(ctx, M, "CG", b, E=1e-10)
    assert ctx.solve_kernel() == kernel
    assert r.converged and r.true_rel_res < 1e-9, (r.status, r.true_rel_res)
    M.close()


def skew(A):
    """The pattern of A with 1 above, -1 below and 0 on the diagonal; where A's
    diagonals hold different values, 2 and -2 between rows 0 and 1."""
    row = np.repeat(np.arange(A.n), np.diff(A.ptr))
    val = np.sign(A.col - row).astype(float)
    if np.unique(A.val).size > 2:
        val[(row + A.col == 1)] *= 2.0
    return CSR(A.ptr, A.col, val)


@pytest.mark.parametrize("rhs", ["breakdown", "zero"])
@pytest.mark.parametrize("name", sorted(SYSTEMS))
def test_breakdown_and_zero_rhs(ks, ctx, name, rhs):
    kernel, make = SYSTEMS[name]
    A = skew(make()) if rhs == "breakdown" else make()
    M = ctx.matrix(A)
    b = np.ones(A.n) if rhs == "breakdown" else np.zeros(A.n)
    got = ks.solve(ctx, M, "CG", b, E=1e-10, L=100)
    served = ctx.solve_kernel()
    want = ks.solve(ctx, M, "CG", b, E=1e-10, L=100, cluster_solve=1)
    M.close()
    assert served == kernel
    assert got.status == want.status == (3 if rhs == "breakdown" else 4)  # KS_BREAKDOWN, KS_NAN_DETECTED
    assert got.loop == want.loop and np.array_equal(got.hist_err, want.hist_err, equal_nan=True)
    assert np.array_equal(got.hist_iter, want.hist_iter)
    assert not got.x.any() and not want.x.any()
