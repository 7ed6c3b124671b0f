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


@pytest.mark.parametrize("degree,graphs", [(80, 3), (216, 1)])
def test_kept_weights_have_a_limit(cuda, degree, graphs):
    """Graphs of 100 M edges, whose weights take 0.4 GB each, and one whose weights alone exceed the limit of a gigabyte."""
    import cxgnncomp_backend as be
    n = 1_250_000
    be.forget_graphs()
    gen = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(n, 384, device="cuda", generator=gen).to(torch.bfloat16).requires_grad_(True)
    g = torch.randn(n, 384, device="cuda", generator=gen).to(torch.bfloat16)
    ptr = torch.arange(n + 1, device="cuda") * degree
    ids = [torch.randint(0, n, (n * degree,), device="cuda", generator=gen, dtype=torch.int32) for _ in range(graphs)]

    def gradient(idx):
        return torch.autograd.grad(be.sage_mean_forward(x, ptr, idx, n), [x], g)[0]

    gradient(ids[0])  # grows the stream's scratch
    be.forget_graphs()
    start = torch.cuda.memory_allocated()
    be._transposed_graph(ptr, ids[0], n, n)
    one = torch.cuda.memory_allocated() - start  # a transposed graph without weights
    be.forget_graphs()
    first = [gradient(idx) for idx in ids]
    kept = torch.cuda.memory_allocated() - start - sum(t.numel() * 2 for t in first) - graphs * one
    assert len(be._TRANSPOSE_CACHE) == graphs
    assert abs(kept - (2 * 4 * n * degree if graphs > 1 else 0)) < 32 << 20  # blocks are cut to a megabyte
    for want, idx in zip(first, ids):  # weights that have made room are made again
        assert torch.equal(gradient(idx), want)
    be.forget_graphs()
