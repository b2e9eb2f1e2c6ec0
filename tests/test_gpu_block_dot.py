"""GPU: the block dot with one and with two elements of a vector in flight
(block_dot_pair; ks_block_dot_noalloc's own rule).

Both add a thread's terms in the same order on the same grid, so a projection's
bits must not depend on how many others are taken with it; against FP64 torch the
error of a sum of n terms of N(0, 1) products is below n eps times the largest
partial sum, far inside 1e-11 |v| |w|.
"""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def vectors(n, k):
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(n + k)
    V = torch.randn(k, n, generator=g, device="cuda", dtype=torch.float64)
    w = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    return V, w


def project(ks, ctx, V, w, k, noalloc):
    import torch

    n = w.numel()
    h = torch.full((k,), float("nan"), device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    if noalloc:
        s = torch.cuda.Stream()
        assert ks.lib().ks_block_dot_noalloc(C.c_void_p(V.data_ptr()), n, k, C.c_void_p(w.data_ptr()), n,
                                             C.c_void_p(h.data_ptr()), C.c_void_p(s.cuda_stream)) == 0
    else:
        wrap = lambda t: ks.Vector(ctx, n=t.numel(), wrap_ptr=t.data_ptr())  # noqa: E731
        Vv, wv = wrap(V), wrap(w)
        ks.block_dot(Vv, n, k, wv, out_device_ptr=h.data_ptr())
        ctx.synchronize()
    torch.cuda.synchronize()
    return h


# rows around the rules' limits (606,208 = four elements per thread; 120 MB of
# vectors), odd ones, and ones that leave threads with 4 and 5 elements
@pytest.mark.parametrize("noalloc", [False, True])
@pytest.mark.parametrize("n,k", [(606207, 25), (606208, 25), (606209, 24), (606209, 30), (700001, 24), (1000003, 17),
                                 (1000003, 40), (2097152, 19), (1700001, 8), (1700001, 9), (4096000, 5)])
def test_same_bits_with_fewer_vectors(ks, ctx, n, k, noalloc):
    import torch

    V, w = vectors(n, k)
    h = project(ks, ctx, V, w, k, noalloc)
    bound = 1e-11 * V.norm(dim=1) * w.norm()
    assert bool(((h - V @ w).abs() <= bound).all())
    for m in (1, 2, 8, 15, 16):
        if m < k:
            assert torch.equal(project(ks, ctx, V, w, m, noalloc), h[:m]), m


CAPTURE = """
import ctypes as C, sys
import torch
sys.path.insert(0, sys.argv[1])
import solver_cpp_b200 as ks
L = ks.lib()
n, k = 1000003, 24
V = torch.randn(k, n, device="cuda", dtype=torch.float64)
w = torch.randn(n, device="cuda", dtype=torch.float64)
h = torch.zeros(k, device="cuda", dtype=torch.float64)
p = lambda t: C.c_void_p(t.data_ptr())
s = torch.cuda.Stream()
torch.cuda.synchronize()
call = lambda n, k: L.ks_block_dot_noalloc(p(V), V.shape[1], k, p(w), n, p(h), C.c_void_p(s.cuda_stream))
assert call(1000, 1) == 0  # the first call; a captured one may take the other kernel
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g, stream=s):
    assert call(n, k) == 0
h.fill_(float("nan"))
g.replay()
torch.cuda.synchronize()
bound = 1e-11 * V.norm(dim=1) * w.norm()
assert bool(((h - V @ w).abs() <= bound).all())
want = h.clone()
assert call(n, k) == 0
torch.cuda.synchronize()
assert torch.equal(h, want)
print("captured")
"""


def test_noalloc_under_capture_after_a_first_small_call():
    """In a process of its own: the captured call is the first to take its kernel."""
    import os
    import subprocess
    import sys

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CAPTURE, root], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "captured" in r.stdout, r.stderr[-2000:]
