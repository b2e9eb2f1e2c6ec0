"""GPU: host time of a solve call beside the solve itself."""
import time

import numpy as np
import pytest

from test_gpu_tile_cg import constant_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 66000, 3), (3, 250000, 3)])
def test_long_boxes(ks, ctx, shape):
    """The search for a tile must not go through every height of a long box: a
    solve of no iterations takes less than 0.4 ms (the best of ten; 0.2 ms on
    boxes of the same size that are long in z)."""
    A = constant_box(shape)
    M = ctx.matrix(A)
    b, x = ctx.vector(np.ones(A.n)), ctx.vector(n=A.n)
    took = []
    for _ in range(10):
        t0 = time.perf_counter()
        ks.solve(ctx, M, "CG", b, x=x, E=1e-14, L=0)
        took.append(time.perf_counter() - t0)
    M.close()
    assert min(took) < 4e-4, min(took)
