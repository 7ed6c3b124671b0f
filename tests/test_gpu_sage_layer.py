"""The SAGE layer as one operator against its parts in float64: the mean before and behind the product, fewer destinations
than sources, widths that the products take themselves and such that go to torch in the backward."""
import pytest
import torch

from helpers import randn, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,n_out", [(100, 256), (256, 47), (16, 16), (300, 64), (64, 5)])
@pytest.mark.parametrize("n_src,n_dst", [(700, 700), (900, 130), (50, 1)])
@pytest.mark.parametrize("bias", [True, False])
def test_layer(cuda, k, n_out, n_src, n_dst, bias):
    import cxgnncomp
    import cxgnncomp_backend as be
    gen = torch.Generator().manual_seed(k + n_dst)
    deg = torch.randint(0, 7, (n_dst,), generator=gen)
    deg[0] = 3
    ptr = torch.cat([torch.zeros(1, dtype=torch.int64), deg.cumsum(0)])
    idx = torch.randint(0, n_src, (int(ptr[-1]),), generator=gen)
    conv = cxgnncomp.MySageConv(k, n_out, bias=bias).cuda()
    x = randn((n_src, k), 1)
    g = randn((n_dst, n_out), 2)
    xd = x.cuda().requires_grad_()
    p = ptr.cuda(), idx.cuda()
    assert be.sage_layer(xd, *p, conv.lin_l.weight, conv.lin_r.weight, conv.lin_l.bias, n_dst, k <= n_out) is not None
    y = conv(xd, *p, n_dst)
    got = torch.autograd.grad(y, [xd, *conv.parameters()], g.cuda())
    ref = [t.detach().cpu().double().requires_grad_() for t in (xd, *conv.parameters())]
    w = dict(zip([name for name, _ in conv.named_parameters()], ref[1:]))
    dst = torch.repeat_interleave(torch.arange(n_dst), deg)
    mean = torch.zeros(n_dst, k, dtype=torch.float64).index_add(0, dst, ref[0][idx]) / deg.clamp(min=1).unsqueeze(1)
    want = mean @ w["lin_l.weight"].t() + ref[0][:n_dst] @ w["lin_r.weight"].t()
    if bias:  # the mean of no neighbours is zero, also of a transformed and shifted one
        want = want + (w["lin_l.bias"] if k <= n_out else w["lin_l.bias"] * (deg > 0).unsqueeze(1))
    assert rel_err(y.detach().cpu(), want.detach()) < 3e-6
    with torch.no_grad():
        assert rel_err(conv(xd, *p, n_dst).cpu(), want.detach()) < 3e-6
    for a, b in zip(got, torch.autograd.grad(want, ref, g.double())):
        assert a.shape == b.shape and rel_err(a.cpu(), b) < 5e-6
