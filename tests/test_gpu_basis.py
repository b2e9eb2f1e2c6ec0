"""GPU: the block AXPY (basis_kernel) at the edges of its launch shapes.

Every element's chain w -= h_i v_i rounds the product and the difference one
after the other, in index order: the same bits as the separate products and
differences of FP64 torch.
"""
import pytest

pytestmark = pytest.mark.gpu

# one element per thread in one wave (up to 592 CTAs of 256: 151,552 rows), in
# more CTAs (303,104; from 64 vectors any), two per thread and a rest
ROWS = [1, 255, 257, 151551, 151552, 151553, 303104, 303105, 400001, 606209, 700001]
VECTORS = [1, 7, 8, 9, 17, 63, 64, 65]


@pytest.mark.parametrize("n", ROWS)
def test_block_axpy_bits(ks, ctx, n):
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    K = max(VECTORS)
    V = torch.randn(K, n, generator=g, device="cuda", dtype=torch.float64)
    w0 = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    h = torch.randn(K, generator=g, device="cuda", dtype=torch.float64)
    hh = h.cpu().tolist()
    Vv = ks.Vector(ctx, n=V.numel(), wrap_ptr=V.data_ptr())
    want = w0.clone()
    for k in range(1, K + 1):
        want = want - V[k - 1] * hh[k - 1]
        if k not in VECTORS:
            continue
        w = w0.clone()
        torch.cuda.synchronize()
        wv = ks.Vector(ctx, n=n, wrap_ptr=w.data_ptr())
        ks.block_axpy(Vv, n, k, h.data_ptr(), wv)
        ctx.synchronize()
        assert torch.equal(w, want), k
