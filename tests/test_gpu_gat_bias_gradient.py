"""The gradients of a GAT layer with joined heads where the set-up of the backward pass also sums the columns of dy: one, two and
four columns per lane and one, two and four rounds of them, rows that are no multiple of a warp's or a block's share, more tiles
than are walked at once. Against float64; 2e-5 as in the other tests of the layer, and for the bias, whose gradient is a plain
sum, 1e-6: n terms added in fp32 by up to 1,184 * 8 warps, 2^-24 * sqrt(n / 9,472) of random rounding and the joins' few steps."""
import pytest
import torch

from helpers import random_csr, randn, rel_err
from test_gpu_gat_layer import reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,c,n", [(1, 32, 7), (2, 16, 33), (4, 16, 1000), (1, 64, 31), (4, 32, 257), (8, 16, 1), (8, 32, 400), (2, 128, 63),
                                   (8, 64, 130), (4, 128, 301), (4, 16, 40000)])
def test_gradients(cuda, h, c, n):
    import cxgnncomp_backend as be
    ptr, idx = random_csr(n, n + 3, 9, seed=h * c, hub=500)
    args = [randn((n + 3, h, c), 1), randn((1, h, c), 2) * 0.3, randn((1, h, c), 3) * 0.3, randn((h * c,), 4)]
    g = randn((n, h * c), 5)
    dev = [t.cuda().requires_grad_() for t in args]
    ref = [t.double().requires_grad_() for t in args]
    y = be.gat_layer(*dev, ptr.cuda(), idx.cuda(), n, 0.2, True)
    want = reference(*ref, ptr, idx, n, 0.2, True)
    got = torch.autograd.grad(y, dev, g.cuda())
    exp = torch.autograd.grad(want, ref, g.double())
    for a, b in zip(got[:3], exp[:3]):
        assert a.shape == b.shape and rel_err(a.cpu(), b) < 2e-5
    assert rel_err(got[3].cpu(), exp[3]) < 1e-6
