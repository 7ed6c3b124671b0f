"""A GAT layer behind its linear transform as one operator against the separate operators and float64: head widths that are
and are not whole vectors, heads joined and averaged, fewer destinations than sources, empty rows."""
import pytest
import torch

from helpers import randn, rel_err

pytestmark = pytest.mark.gpu


def reference(x, att_s, att_d, bias, ptr, idx, n, slope, concat):
    h, c = x.shape[1:]
    deg = ptr[1:] - ptr[:-1]
    dst = torch.repeat_interleave(torch.arange(n), deg)
    e = torch.nn.functional.leaky_relu((x * att_s).sum(-1)[idx] + (x * att_d).sum(-1)[dst], slope)
    p = torch.exp(e - e.max())
    den = torch.zeros(n, h, dtype=x.dtype).index_add(0, dst, p).clamp(min=1e-300)
    y = torch.zeros(n, h, c, dtype=x.dtype).index_add(0, dst, (p / den[dst]).unsqueeze(-1) * x[idx])
    y = y.reshape(n, h * c) if concat else y.mean(1)
    return y if bias is None else y + bias


@pytest.mark.parametrize("h,c,concat", [(4, 32, True), (2, 64, False), (1, 128, True), (8, 4, True), (4, 2, False), (16, 1, True),
                                        (2, 8, False)])
@pytest.mark.parametrize("n_src,n_dst", [(40, 40), (900, 517)])
@pytest.mark.parametrize("with_bias", [True, False])
def test_layer(cuda, h, c, concat, n_src, n_dst, with_bias):
    import cxgnncomp_backend as be
    gen = torch.Generator().manual_seed(h * c + n_dst)
    deg = torch.randint(0, 9, (n_dst,), generator=gen)
    deg[1] = 0
    ptr = torch.cat([torch.zeros(1, dtype=torch.int64), deg.cumsum(0)])
    idx = torch.randint(0, n_src, (int(ptr[-1]),), generator=gen)
    width = h * c if concat else c
    args = [randn((n_src, h, c), 1), randn((1, h, c), 2) * 0.3, randn((1, h, c), 3) * 0.3,
            randn((width,), 4) if with_bias else None]
    g = randn((n_dst, width), 5)
    dev = [None if t is None else t.cuda().requires_grad_() for t in args]
    ref = [None if t is None else t.double().requires_grad_() for t in args]
    assert be.gat_layer_supported(*dev)
    y = be.gat_layer(*dev, ptr.cuda(), idx.cuda(), n_dst, 0.2, concat)
    want = reference(*ref, ptr, idx, n_dst, 0.2, concat)
    assert rel_err(y.detach().cpu(), want.detach()) < 1e-5
    with torch.no_grad():
        assert torch.equal(be.gat_layer(*dev, ptr.cuda(), idx.cuda(), n_dst, 0.2, concat), y)
    given = [i for i in range(4) if dev[i] is not None]
    got = torch.autograd.grad(y, [dev[i] for i in given], g.cuda())
    exp = torch.autograd.grad(want, [ref[i] for i in given], g.double())
    for a, b in zip(got, exp):
        assert a.shape == b.shape and rel_err(a.cpu(), b) < 2e-5


@pytest.mark.parametrize("h,c", [(1, 3), (3, 47), (4, 47), (1, 4), (5, 12), (4, 100), (1, 132), (2, 256)])
def test_scores_and_mean(cuda, h, c):
    import cxgnncomp_backend as be
    for n in (1, 300, 5000):
        x, s, d, b = randn((n, h, c), n), randn((1, h, c), 2), randn((1, h, c), 3), randn((c,), 4)
        a_s, a_d = be.gat_scores(x.cuda(), s.cuda(), d.cuda(), (n + 1) // 2)
        assert rel_err(a_s.cpu(), (x.double() * s.double()).sum(-1)) < 2e-6
        assert rel_err(a_d.cpu(), (x.double() * d.double()).sum(-1)[:(n + 1) // 2]) < 2e-6
        assert rel_err(be._native.head_mean_bias(x.cuda(), b.cuda(), h, c).cpu(), x.double().mean(1) + b.double()) < 2e-6


@pytest.mark.parametrize("h,c", [(4, 17), (4, 21), (4, 30), (16, 5), (16, 15), (8, 27), (8, 41), (4, 47), (4, 63), (2, 62)])
def test_vectors_across_heads(cuda, h, c):
    import cxgnncomp_backend as be
    gen = torch.Generator().manual_seed(h * c)
    n = 600
    deg = torch.randint(0, 9, (n,), generator=gen)
    deg[5] = 9000  # cut by many tiles
    ptr = torch.cat([torch.zeros(1, dtype=torch.int64), deg.cumsum(0)])
    idx = torch.randint(0, n, (int(ptr[-1]),), generator=gen)
    args = [randn((n, h, c), 1), randn((1, h, c), 2) * 0.3, randn((1, h, c), 3) * 0.3, randn((c,), 4)]
    with torch.no_grad():
        got = be.gat_layer(*[t.cuda() for t in args], ptr.cuda(), idx.cuda(), n, 0.2, False)
    assert rel_err(got.cpu(), reference(*[t.double() for t in args], ptr, idx, n, 0.2, False)) < 1e-5
