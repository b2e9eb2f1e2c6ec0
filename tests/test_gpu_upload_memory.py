"""GPU: what an uploaded matrix keeps in device memory.

The sliced copy for the one-launch CG of CSR matrices holds up to twice the FP64
values and offsets: it is kept only where that kernel can run.
"""
import numpy as np
import pytest

from solver_cpp_b200.matrices import poisson3d
from test_gpu_csr_cg import graph

pytestmark = pytest.mark.gpu

MB = 1 << 20


def kept(ctx, A, **kw):
    """Device bytes an upload keeps, and what CSR with both index forms takes."""
    import torch

    ctx.matrix(A, **kw).close()  # the context's own allocations
    ctx.synchronize()
    free = torch.cuda.mem_get_info()[0]
    M = ctx.matrix(A, **kw)
    ctx.synchronize()
    used = free - torch.cuda.mem_get_info()[0]
    M.close()
    # values, int32 and int16 columns, row offsets, row blocks; 2 MB per allocation for its granularity
    return used, A.nnz * 14 + A.n * 8 + 12 * MB


def test_slices_are_kept_where_the_window_fits(ctx):
    A = graph(250000, 6000, 6000, 40)
    used, csr = kept(ctx, A)
    assert used > csr + 8 * A.nnz


@pytest.mark.parametrize("case", ["window", "no_diag"])
def test_no_slices_where_nothing_reads_them(ks, ctx, case):
    """Offsets wider than shared memory; KS_MAT_NO_DIAG, which keeps CSR only."""
    A, kw = (graph(250000, 16000, 16000, 40), {}) if case == "window" else (poisson3d(84, 84, 84), dict(diag=False))
    used, csr = kept(ctx, A, **kw)
    assert used <= csr, (used, csr)
    M = ctx.matrix(A, **kw)
    ks.solve(ctx, M, "CG", np.ones(A.n), E=1e-14, L=2)
    assert ctx.solve_kernel() == ""
    M.close()
