"""The fp32 linear transform on the tensor cores at the edges of its tiles (128 rows, 32 columns of K, blocks of columns of
the result), with bias, a matrix to add and all gradients, against float64; and the shapes that go to torch."""
import pytest
import torch

from helpers import randn, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n", [(1, 4, 1), (1, 32, 16), (127, 16, 17), (128, 36, 47), (129, 48, 64), (300, 100, 256),
                                   (1000, 128, 128), (20000, 128, 188), (500, 256, 47), (700, 300, 20), (257, 1084, 40),
                                   (64, 64, 1000), (40, 33, 8), (40, 2048, 8)])
@pytest.mark.parametrize("bias,add", [(False, False), (True, True), (False, True)])
def test_linear(cuda, m, k, n, bias, add):
    import cxgnncomp_backend as be
    args = [randn((m, k), m + k), randn((n, k), n) * 0.1, randn((n,), 3) if bias else None, randn((m, n), 4) if add else None]
    g = randn((m, n), 5)
    dev = [None if t is None else t.cuda().requires_grad_() for t in args]
    ref = [None if t is None else t.double().requires_grad_() for t in args]
    y = be.linear(*dev)
    want = torch.nn.functional.linear(*ref[:3]) + (ref[3] if add else 0)
    assert rel_err(y.detach().cpu(), want.detach()) < 2e-6
    with torch.no_grad():
        assert torch.equal(be.linear(*dev), y)
    assert rel_err(be.linear(*dev, same_bits=True).detach().cpu(), want.detach()) < 2e-6
    given = [i for i in range(4) if dev[i] is not None]
    got = torch.autograd.grad(y, [dev[i] for i in given], g.cuda())
    exp = torch.autograd.grad(want, [ref[i] for i in given], g.double())
    for a, b in zip(got, exp):
        assert a.shape == b.shape and rel_err(a.cpu(), b) < 4e-6
