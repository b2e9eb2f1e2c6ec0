"""GPU: k_cg_tile (ks_tile_cg.cuh), CG of constant-coefficient boxes on tiles of
lines, against the kernel-per-step engine.

Element operations are the engine's and only the dot products add their terms in
another order. The systems are diagonally dominant by 5 %, so the histories and
solutions of the first iterations agree to 1e-9 (as in test_gpu_chip_cg.py).

Which tile a box gets: by lines and bz planes as named below (148 SMs, 227 KB of
shared memory per CTA). A thread works on blocks of 8 planes, so what can go
wrong lies at bz mod 8, at last tiles thinner than the others, and at boxes that
are one tile high or deep.
"""
import numpy as np
import pytest

from solver_cpp_b200.matrices import poisson3d
from test_gpu_chip_cg import agree

pytestmark = pytest.mark.gpu

SHAPES = [
    (67, 56, 162),    # by 7, bz 9: a block of one plane
    (46, 14, 1261),   # bz 18, the last tile one plane
    (113, 113, 113),  # bz 11, the last tile 3 planes
    (315, 241, 8),    # by 4, the last one line; bz 4: less than a block
    (117, 117, 117),  # bz 13
    (124, 124, 124),  # bz 14
    (21, 111, 261),   # bz 15
    (9, 300, 301),    # by 43; the last tile one plane
    (311, 3, 784),    # one tile in y
    (158, 1284, 3),   # one tile in z, of three planes
    (3, 848, 924),    # by 170, bz 32: 2.35M rows
]


def constant_box(shape, skew=0.0):
    """-1 beside a dominant diagonal; with skew every diagonal has a value of its own."""
    A = poisson3d(*shape)
    off = A.col - np.repeat(np.arange(A.n), np.diff(A.ptr))
    for k, o in enumerate(np.unique(off)):
        A.val[off == o] = 6.3 if o == 0 else -1.0 + skew * (k - 3)
    return A


def both(ks, ctx, A, b=None, **kw):
    """The solve on tiles and kernel by kernel."""
    M = ctx.matrix(A)
    b = np.random.default_rng(1).standard_normal(A.n) if b is None else b
    tile = ks.solve(ctx, M, "CG", b, cluster_solve=0, **kw)
    assert ctx.solve_kernel() == "k_cg_tile"
    step = ks.solve(ctx, M, "CG", b, cluster_solve=1, **kw)
    assert ctx.solve_kernel() == ""
    M.close()
    return tile, step


@pytest.mark.parametrize("shape", SHAPES)
def test_against_engine(ks, ctx, shape):
    agree(*both(ks, ctx, constant_box(shape), E=1e-14, L=30))


@pytest.mark.parametrize("shape", [(93, 91, 90), (113, 113, 113), (131, 62, 77)])
def test_unsymmetric_constants(ks, ctx, shape):
    """Seven different values, A not its transpose: each neighbour takes its own."""
    agree(*both(ks, ctx, constant_box(shape, skew=0.01), E=1e-14, L=15))


@pytest.mark.parametrize("L", [0, 1, 2])
def test_stops_at_maxloop(ks, ctx, L):
    agree(*both(ks, ctx, constant_box((93, 91, 90)), E=1e-14, L=L))


def test_converges(ks, ctx):
    tile, step = both(ks, ctx, constant_box((113, 113, 113)), E=1e-9)
    assert tile.converged and tile.true_rel_res < 2e-9
    agree(tile, step)


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("diagonal", [0, 5])
def test_constants_that_are_not_finite(ks, ctx, value, diagonal):
    """An entry a row does not have must not count: inf times the zero beside the
    box would be NaN."""
    A = constant_box((93, 91, 90))
    off = A.col - np.repeat(np.arange(A.n), np.diff(A.ptr))
    A.val[off == np.unique(off)[diagonal]] = -value
    M = ctx.matrix(A)
    chip, step = [ks.solve(ctx, M, "CG", np.ones(A.n), E=1e-14, L=10, cluster_solve=c) for c in (0, 1)]
    M.close()
    assert chip.status == step.status and chip.loop == step.loop, (chip.status, step.status, chip.loop, step.loop)
    assert np.array_equal(chip.hist_err, step.hist_err, equal_nan=True)
