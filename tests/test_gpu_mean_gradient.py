"""Gradient of a mean aggregation: by weights per transposed edge or by a pass over the incoming gradient, whichever the sizes choose,
against float64; weights that one stream has made and another uses; 3-D features."""
import pytest
import torch

from helpers import random_csr, randn

pytestmark = pytest.mark.gpu


def _check(ptr, idx, n_src, shape, dtype):
    import cxgnncomp_backend as be
    n = ptr.shape[0] - 1
    x = randn((n_src, *shape), 1).to(dtype).cuda().requires_grad_(True)
    g = randn((n, *shape), 2).to(dtype).cuda()
    y = be.sage_mean_forward(x, ptr.cuda(), idx.cuda(), n)
    (dx,) = torch.autograd.grad(y, [x], g)
    deg = (ptr[1:] - ptr[:-1])
    dst = torch.repeat_interleave(torch.arange(n), deg)
    w = g.double().cpu() / deg.clamp(min=1).double().view(-1, *([1] * len(shape)))
    want = torch.zeros(n_src, *shape, dtype=torch.float64).index_add_(0, idx, w[dst])
    assert dx.dtype == dtype
    # one rounding of 1 / degree, one per product, sequential sums of at most a few hundred terms; bf16: the scaled gradient
    # (where a pass scales it) and the result are rounded to eight bits
    assert (dx.double().cpu() - want).norm() <= (1e-6 if dtype == torch.float32 else 2 ** -8) * want.norm()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("deg,shape", [(3, (64,)), (3, (47,)), (60, (4,)), (60, (64,)), (20, (1,)), (5, (2, 16))])
@pytest.mark.parametrize("n", [300, 9000])
def test_gradient(cuda, dtype, deg, shape, n):
    ptr, idx = random_csr(n, n - 50, deg, seed=deg + n, hub=150)
    _check(ptr, idx, n - 50, shape, dtype)


def test_other_streams(cuda):
    import cxgnncomp_backend as be
    be.forget_graphs()
    n = 4000
    ptr, idx = (t.cuda() for t in random_csr(n, n, 4, seed=1))
    x, g = randn((n, 64), 1).cuda().requires_grad_(True), randn((n, 64), 2).cuda()

    def gradient():
        return torch.autograd.grad(be.sage_mean_forward(x, ptr, idx, n), [x], g)[0]

    torch.cuda.synchronize()
    first = gradient()
    others = []
    for _ in range(3):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            others.append(gradient())
    torch.cuda.synchronize()
    assert all(torch.equal(first, o) for o in others)
    be.forget_graphs()
    assert torch.equal(first, gradient())
