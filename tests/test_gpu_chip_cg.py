"""GPU: CG with the matrix on chip (ks_chip_cg.cuh), FP64 whole solves and the
FP32 / BF16-valued inner CG, against the kernel-per-step engine.

Both apply the same operations to every element and differ only in the order
in which the dot products add their terms. Over the first 40 iterations of
these well-conditioned systems (diagonally dominant by 5 %, so a relative
rounding difference of 1e-16 per sum grows by a few orders at most) the
histories and solutions therefore agree to 1e-9; the inner solve's
coefficients are rounded to FP32, which absorbs the difference: there the two
paths agree bit for bit.
"""
import numpy as np
import pytest

from solver_cpp_b200.matrices import CSR

pytestmark = pytest.mark.gpu


def banded(n, offsets, seed=0, keep=None, skew=0.0):
    """Matrix with entries at the given offsets (0 among them, ascending):
    random symmetric values, `skew` added to the upper ones, a dominant
    diagonal; keep(i, off) drops entries."""
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    has = np.zeros((n, len(offsets)), dtype=bool)
    val = np.zeros((n, len(offsets)))
    up = {o: -rng.uniform(0.5, 1.0, n) for o in offsets if o > 0}
    for d, o in enumerate(offsets):
        has[:, d] = (i + o >= 0) & (i + o < n)
        if keep is not None and o:
            lo = np.minimum(i, i + o)
            has[:, d] &= keep(np.maximum(lo, 0), abs(o))
        if o > 0:
            val[:, d] = up[o] + skew
        elif o < 0:
            val[:, d] = np.roll(up[-o], -o) if -o in up else -0.3
    val *= has
    d0 = offsets.index(0)
    val[:, d0] = 1.05 * np.abs(val).sum(1) + 0.1
    cols = i[:, None] + np.asarray(offsets)
    ptr = np.zeros(n + 1, dtype=np.int32)
    ptr[1:] = np.cumsum(has.sum(1))
    return CSR(ptr, cols[has].astype(np.int32), val[has])


def box(nx, ny, nz=1, seed=0, wrap=False, skew=0.0):
    """5- or 7-point stencil on a box; wrap keeps the entries across the ends
    of lines and planes (no box then: the run-of-rows layout)."""
    offs = [-nx, -1, 0, 1, nx] if nz == 1 else [-nx * ny, -nx, -1, 0, 1, nx, nx * ny]

    def inside(i, o):
        return (i % nx < nx - 1) if o == 1 else (((i // nx) % ny < ny - 1) if o == nx else np.ones(len(i), bool))

    return banded(nx * ny * nz, offs, seed, None if wrap else inside, skew)


# runs of rows (2D): 8,193 rows is the smallest system of this path, 16,384 =
# 32 CTAs of 512, 16,385 one row more, 65,536 the largest on 32 CTAs, 65,537
# the smallest on one CTA per SM, 606,208 = 148 x 4,096 the largest
RUNS = [(8193, 1), (128, 128), (145, 113), (256, 256), (65537, 1), (333, 331), (700, 701), (1024, 592)]
# tiles of lines (3D): edges that the tile does and does not divide, single
# lines, planes thinner than a tile, flat and long boxes, and boxes near the limit
BOXES = [(21, 20, 20), (32, 16, 32), (37, 41, 43), (7, 200, 9), (300, 5, 11), (2, 90, 91), (64, 64, 64), (81, 81, 81)]


def both(ks, ctx, A, seed=1, L=40):
    M = ctx.matrix(A)
    b = np.random.default_rng(seed).standard_normal(A.n)
    chip = ks.solve(ctx, M, "CG", b, E=1e-14, L=L, cluster_solve=0, profile=1)
    step = ks.solve(ctx, M, "CG", b, E=1e-14, L=L, cluster_solve=1)
    M.close()
    return chip, step


def agree(chip, step):
    assert chip.status == step.status and chip.loop == step.loop, (chip.status, step.status, chip.loop, step.loop)
    assert np.array_equal(chip.hist_iter, step.hist_iter)
    assert np.allclose(chip.hist_err, step.hist_err, rtol=1e-9, atol=0)
    assert np.linalg.norm(chip.x - step.x) <= 1e-9 * np.linalg.norm(step.x)


@pytest.mark.parametrize("shape", RUNS + BOXES)
def test_fp64_cg_against_engine(ks, ctx, shape):
    A = box(*shape) if shape[1] > 1 else banded(shape[0], [-1, 0, 1])
    chip, step = both(ks, ctx, A)
    assert chip.report["n_mv"] == 1 and chip.report["n_dot"] == 0, chip.report
    agree(chip, step)


@pytest.mark.parametrize("offsets", [[-700, -3, 0, 3, 700], [-5, -2, 0, 4], [-40, -30, -20, -10, 0, 10, 20, 30],
                                     [-1500, -37, -1, 0, 1, 37, 1500]])
def test_fp64_cg_any_offsets(ks, ctx, offsets):
    """Any diagonals, in runs of rows; unsymmetric values keep the full layout."""
    chip, step = both(ks, ctx, banded(21000, offsets, skew=0.01), L=15)
    assert chip.report["n_mv"] == 1 and chip.report["n_dot"] == 0, chip.report
    agree(chip, step)


def test_fp64_cg_box_with_wrapped_entries(ks, ctx):
    """A 7-diagonal matrix with entries across line ends is no box."""
    chip, step = both(ks, ctx, box(31, 29, 23, wrap=True))
    agree(chip, step)


def test_fp64_cg_unsymmetric_box(ks, ctx):
    chip, step = both(ks, ctx, box(31, 29, 23, skew=0.02), L=15)
    agree(chip, step)


@pytest.mark.parametrize("L", [0, 1, 2])
def test_fp64_cg_stops_at_maxloop(ks, ctx, L):
    chip, step = both(ks, ctx, box(101, 97), L=L)
    agree(chip, step)


@pytest.mark.parametrize("prec", ["fp32", "bf16"])
@pytest.mark.parametrize("shape", [(11, 10, 9), (16, 16, 2), (37, 41, 43), (130, 127), (81, 80, 79), (99, 99, 99),
                                   (1100, 1101)])
def test_inner_cg_bitwise(ks, ctx, shape, prec):
    """VPCG with the inner CG on chip and kernel by kernel: the same bits."""
    A = box(*shape)
    M = ctx.matrix(A, fp32=prec == "fp32", bf16=prec == "bf16")
    b = np.random.default_rng(3).standard_normal(A.n)
    kw = dict(inner="CG", E=1e-11, L=4, l=20, e=1e-30, inner_precision=prec)
    chip = ks.solve(ctx, M, "VPCG", b, inner_fast=0, **kw)
    step = ks.solve(ctx, M, "VPCG", b, inner_fast=1, **kw)
    M.close()
    assert chip.status == step.status and np.array_equal(chip.hist_err, step.hist_err)
    assert np.array_equal(chip.x, step.x)


def test_inner_cg_of_another_length(ks, ctx):
    """A second solve on the same context reuses the published array with new
    tags; an inner solve that stops early leaves the same state."""
    A = box(37, 41, 43)
    M = ctx.matrix(A, fp32=True)
    b = np.random.default_rng(3).standard_normal(A.n)
    for l, e in ((20, 1e-30), (3, 1e-30), (50, 1e-2)):
        kw = dict(inner="CG", E=1e-10, L=60, l=l, e=e, inner_precision="fp32")
        chip = ks.solve(ctx, M, "VPCG", b, inner_fast=0, **kw)
        step = ks.solve(ctx, M, "VPCG", b, inner_fast=1, **kw)
        assert chip.status == step.status == 0 and np.array_equal(chip.x, step.x)
    M.close()


# boxes whose matrix does not fit on chip (k_cg_tile): tiles that divide the
# box and ones that do not, long and short lines, the largest that fit
TILES64 = [(91, 90, 89), (128, 128, 128), (130, 127, 129), (300, 60, 61), (9, 300, 301), (1200, 40, 33)]


@pytest.mark.parametrize("shape", TILES64)
@pytest.mark.parametrize("const", [False, True])
def test_fp64_tiles_against_engine(ks, ctx, shape, const):
    if const:
        from solver_cpp_b200.matrices import poisson3d

        A = poisson3d(*shape)
        A.val[A.val > 0] = 6.3  # 5 % dominant, as the random ones
    else:
        A = box(*shape)
    chip, step = both(ks, ctx, A, L=30)
    assert chip.report["n_mv"] == 1 and chip.report["n_dot"] == 0, chip.report
    agree(chip, step)


def test_fp64_tiles_unsymmetric_and_with_gaps(ks, ctx):
    """The full layout; and constant values with entries missing inside the box."""
    chip, step = both(ks, ctx, box(93, 91, 90, skew=0.02), L=15)
    agree(chip, step)
    nx, ny, nz = 93, 91, 90

    def some(i, o):
        inside = (i % nx < nx - 1) if o == 1 else (((i // nx) % ny < ny - 1) if o == nx else np.ones(len(i), bool))
        return inside & (i % 7 != 3)

    A = banded(nx * ny * nz, [-nx * ny, -nx, -1, 0, 1, nx, nx * ny], keep=some)
    off = A.val < 0
    A.val[off], A.val[~off] = -1.0, 6.3
    chip, step = both(ks, ctx, A, L=30)
    agree(chip, step)


@pytest.mark.parametrize("prec", ["fp32", "bf16"])
@pytest.mark.parametrize("shape", [(109, 108, 107), (131, 128, 127), (160, 160, 160), (700, 45, 44)])
def test_inner_tiles_bitwise(ks, ctx, shape, prec):
    test_inner_cg_bitwise(ks, ctx, shape, prec)
