"""CPU: the bytes bench.py divides by follow the kernel that ran (constant
diagonals are not read, a matrix held on chip is read once)."""
import numpy as np

from solver_cpp_b200.matrices import convdiff3d, poisson3d, varcoef3d
from test_bench_bytes import _bench


def test_constant_diagonals():
    b = _bench()
    A = poisson3d(7, 6, 5)
    assert b.constant_diagonals(A) and b.constant_diagonals(convdiff3d(5))
    A.val[3] = np.nextafter(A.val[3], 9.0)
    assert not b.constant_diagonals(A) and not b.constant_diagonals(varcoef3d(4))


def test_bytes_of_constant_diagonals():
    b = _bench()
    n, info = 128 ** 3, {"offsets": [-16384, -128, -1, 0, 1, 128, 16384]}
    assert b.spmv_bytes(n, 0, "fp64", 2, 7, 1, constant=1) == 17 * n  # mask, x, y
    assert b.spmv_bytes(n, 0, "fp32", 2, 7, 1, constant=1) == b.spmv_bytes(n, 0, "fp32", 2, 7, 1)
    diff = b.onchip_whole_bytes("CR", n, 7, 1, info, 10) - b.onchip_whole_bytes("CR", n, 7, 1, info, 10, constant=1)
    assert diff == 10 * 4 * 8 * n


def test_bytes_of_a_held_matrix():
    b = _bench()
    n = 512 * 512
    assert b.held_bytes("k_cg_chip", n, "fp64", 5, 1) == n * (3 * 8 + 16)
    assert b.held_bytes("k_cg_chip", n, "bf16", 7, 0) == n * (7 * 2 + 8)
    assert b.held_bytes("k_cg_tile", n, "fp64", 7, 1) == n * 16
    assert b.held_bytes("k_cg_onchip", n, "fp64", 7, 1) is None and b.held_bytes("", n, "fp64", 7, 1) is None
