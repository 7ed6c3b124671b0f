"""The fp32 linear transform of few rows: blocks of 16 columns, fewer, as many and more units of A than the ring holds, and
calls behind one another whose blocks start while the one in front drains. Against float64; 2e-6 is the bound of the
three-term product (six terms kept, cut at 2^-26, sums of up to 2,048 columns), twice that for two in a row."""
import pytest
import torch

from helpers import randn, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n", [(1, 32, 15), (6, 96, 17), (32, 128, 31), (32, 132, 33), (127, 160, 48), (128, 256, 47),
                                   (129, 256, 256), (1100, 100, 256), (1200, 256, 240)])
def test_chain(cuda, m, k, n):
    import cxgnncomp_backend as be
    x, w1, w2, b = randn((m, k), 1), randn((n * 4, k), 2) * 0.1, randn((n, n * 4), 3) * 0.1, randn((n,), 4)
    h = x.double() @ w1.double().t()
    want = h @ w2.double().t() + b.double()
    xd, w1d, w2d, bd = x.cuda(), w1.cuda(), w2.cuda(), b.cuda()
    torch.cuda.synchronize()
    with torch.no_grad():
        for _ in range(3):  # the memory of one round is taken again by the next one
            mid = be.linear(xd, w1d)
            y = be.linear(mid, w2d, bd)
            again = be.linear(mid, w2d, bd, y)
            del mid
    assert rel_err(y.cpu(), want) < 4e-6
    assert rel_err(again.cpu(), 2 * want) < 4e-6
