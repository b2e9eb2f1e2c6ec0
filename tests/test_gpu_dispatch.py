"""GPU: which kernel serves a solve (ks_ctx_solve_kernel).

The on-chip kernels agree with each other and with the engine to rounding, so a
solve that silently took another path would pass every comparison. The shapes
are those of the other test files and the edges of each kernel's range (148 SMs,
227 KB of shared memory per CTA).
"""
import numpy as np
import pytest

from solver_cpp_b200.matrices import convdiff2d, poisson2d, poisson3d, varcoef3d
from test_gpu_chip_cg import banded, box
from test_gpu_csr_cg import graph
from test_gpu_tile_cg import constant_box

pytestmark = pytest.mark.gpu


def gaps(nx, ny, nz):
    """Constant values, some neighbours inside the box missing."""
    def some(i, o):
        inside = (i % nx < nx - 1) if o == 1 else (((i // nx) % ny < ny - 1) if o == nx else np.ones(len(i), bool))
        return inside & (i % 7 != 3)

    A = banded(nx * ny * nz, [-nx * ny, -nx, -1, 0, 1, nx, nx * ny], keep=some)
    off = A.val < 0
    A.val[off], A.val[~off] = -1.0, 6.3
    return A


CG = [
    ("k_cg_resident", lambda: poisson2d(64)),
    ("k_cg_resident", lambda: banded(8192, [-1, 0, 1])),
    ("k_cg_chip", lambda: banded(8193, [-1, 0, 1])),
    ("k_cg_chip", lambda: box(333, 331)),
    ("k_cg_chip", lambda: box(81, 81, 81)),
    ("k_cg_chip", lambda: poisson3d(64, 64, 64)),
    ("k_cg_chip", lambda: banded(148 * 4096, [-1, 0, 1])),
    # the smallest and one of the largest boxes on tiles; boxes whose lines or
    # faces are too long for a tile
    ("k_cg_tile", lambda: constant_box((86, 84, 84))),
    ("k_cg_tile", lambda: constant_box((128, 128, 128))),
    ("k_cg_onchip", lambda: constant_box((130, 127, 129))),
    ("k_cg_onchip", lambda: constant_box((300, 60, 61))),
    ("k_cg_onchip", lambda: constant_box((1200, 40, 33))),
    # more rows than the matrix has room for: other values, entries missing
    ("k_cg_onchip", lambda: box(91, 90, 89)),
    ("k_cg_onchip", lambda: box(93, 91, 90, skew=0.02)),
    ("k_cg_onchip", lambda: gaps(93, 91, 90)),
    ("k_cg_csr", lambda: graph(8193, 3, 3, 2)),
    ("k_cg_csr", lambda: graph(606208, 2000, 2000, 2)),
    ("", lambda: graph(606209, 2000, 2000, 2)),
    ("", lambda: graph(70000, 30000, 30000, 4)),
]


@pytest.mark.parametrize("case", range(len(CG)))
def test_cg(ks, ctx, case):
    kernel, make = CG[case]
    A = make()
    M = ctx.matrix(A)
    b = np.random.default_rng(1).standard_normal(A.n)
    ks.solve(ctx, M, "CG", b, E=1e-14, L=2)
    assert ctx.solve_kernel() == kernel
    ks.solve(ctx, M, "CG", b, E=1e-14, L=2, cluster_solve=1)
    assert ctx.solve_kernel() == ""
    M.close()


@pytest.mark.parametrize("kernel,method,make", [
    ("k_cr_resident", "CR", lambda: poisson2d(64)),
    ("k_cr_onchip", "CR", lambda: poisson3d(40, 40, 40)),
    ("k_bicg_resident", "BICG", lambda: convdiff2d(64)),
    ("k_bicg_onchip", "BICG", lambda: convdiff2d(200)),
    ("", "GMRES", lambda: poisson2d(64)),
    ("k_cg_chip", "VPCG", lambda: varcoef3d(24)),
    ("k_cg_chip", "VPCG", lambda: box(99, 99, 99)),
    ("k_cg_onchip", "VPCG", lambda: box(105, 105, 105)),
    ("k_cg_onchip", "VPCG", lambda: box(109, 108, 107)),
])
def test_other_methods(ks, ctx, kernel, method, make):
    A = make()
    M = ctx.matrix(A, transpose=method == "BICG", fp32=True)
    kw = dict(inner="CG", l=5, e=1e-30, inner_precision="fp32") if method == "VPCG" else {}
    ks.solve(ctx, M, method, np.random.default_rng(1).standard_normal(A.n), E=1e-14, L=2, **kw)
    assert ctx.solve_kernel() == kernel
    M.close()
