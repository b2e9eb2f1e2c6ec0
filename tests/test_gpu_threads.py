"""GPU: solves of several host threads at once, a context each.

The shared memory a kernel may have is set per kernel and device, not per
context: a thread whose system needs less of it must not take the room from
another thread's launch of the same kernel.
"""
import threading

import numpy as np
import pytest

from solver_cpp_b200.matrices import convdiff2d, poisson3d
from test_gpu_csr_cg import graph

pytestmark = pytest.mark.gpu

# two systems of different shared memory on the same kernel, solved in one or two
# iterations, so that launches follow each other closely
PAIRS = {
    "csr": ("CG", lambda: graph(60000, 5000, 5000, 1), lambda: graph(60000, 2500, 2500, 1)),
    "chip": ("CG", lambda: poisson3d(81, 81, 81), lambda: poisson3d(70, 70, 70)),
    "cr": ("CR", lambda: poisson3d(64, 64, 64), lambda: poisson3d(50, 50, 50)),
    "bicg": ("BICG", lambda: convdiff2d(300), lambda: convdiff2d(260)),
}


@pytest.mark.parametrize("name", sorted(PAIRS))
def test_two_threads_on_one_kernel(ks, name):
    method, *make = PAIRS[name]
    mats = [m() for m in make]
    go = threading.Barrier(2)
    errors = []

    def work(A):
        ctx = ks.Context(0)
        try:
            M = ctx.matrix(A, transpose=method == "BICG")
            b = ctx.vector(np.random.default_rng(1).standard_normal(A.n))
            x = ctx.vector(n=A.n)
            ks.solve(ctx, M, method, b, x=x, E=1e-14, L=1)
            want = x.numpy()
            go.wait()
            for _ in range(1200):
                ks.solve(ctx, M, method, b, x=x, E=1e-14, L=1)
            assert np.array_equal(x.numpy(), want)
        except Exception as e:  # noqa: BLE001 (reported by the test's thread)
            errors.append(e)
            go.abort()
        finally:
            ctx.close()

    threads = [threading.Thread(target=work, args=(A,)) for A in mats]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
