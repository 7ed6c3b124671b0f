"""The recorded GAT layer in front of the kink of its LeakyReLU: its features are torch's to the bit, its scores sequential
fp32 multiply-add chains to the bit, and so an edge whose score lies within rounding of zero is on the side on which those
put it, with all gradients."""
import numpy as np
import pytest
import torch

from helpers import randn, rel_err

pytestmark = pytest.mark.gpu


def chain(feat, att):
    """fp32 [n, h]: sum over c of feat * att, one fused multiply-add after the other. The product is exact in 64 bits of
    mantissa, so only a sum that rounds twice onto a tie could differ (2^-40 of all steps)."""
    s = np.zeros(feat.shape[:2], dtype=np.float32)
    f, a = feat.numpy().astype(np.longdouble), att.reshape(feat.shape[1:]).numpy().astype(np.longdouble)
    for j in range(feat.shape[2]):
        s = (f[:, :, j] * a[:, j] + s).astype(np.float32)
    return torch.from_numpy(s)


@pytest.mark.parametrize("h,c", [(1, 4), (4, 32), (3, 12), (8, 36), (2, 64), (16, 4), (5, 100), (1, 33), (4, 47), (2, 7)])
@pytest.mark.parametrize("n", [1, 7, 300, 3001])
def test_scores_in_index_order(cuda, h, c, n):
    import cxgnncomp_backend as be
    x, s, d = randn((n, h, c), n + c), randn((1, h, c), 2), randn((1, h, c), 3)
    n_dst = (n + 1) // 2
    a_s, a_d = be.gat_scores(x.cuda(), s.cuda(), d.cuda(), n_dst)
    assert torch.equal(a_s.cpu(), chain(x, s)) and torch.equal(a_d.cpu(), chain(x, d)[:n_dst])


@pytest.mark.parametrize("heads", [1, 4])
def test_recorded_features_are_torchs(cuda, heads, monkeypatch):
    import cxgnncomp
    import cxgnncomp_backend as be
    seen = []
    name = "gat_layer" if heads > 1 else "sage_sum_forward_edge_value"
    where = be if heads > 1 else cxgnncomp.graph_conv
    real = getattr(where, name)
    monkeypatch.setattr(where, name, lambda x, *args: (seen.append(x), real(x, *args))[1])
    conv = cxgnncomp.MyGATConv(128, 32, heads=heads, concat=True).cuda()
    x = randn((2000, 128), 1).cuda().requires_grad_()
    ptr = torch.arange(0, 4001, 2).cuda()
    idx = torch.randint(0, 2000, (4000,), generator=torch.Generator().manual_seed(2)).cuda()
    conv(x, ptr, idx, 2000, 2000, 4000)
    assert torch.equal(seen[0].reshape(2000, -1), torch.nn.functional.linear(x, conv.lin_src))


def test_scores_next_to_zero(cuda):
    import cxgnncomp
    n, k, h, c = 6000, 64, 4, 16
    torch.manual_seed(10)
    conv = cxgnncomp.MyGATConv(k, c, heads=h, concat=True).cuda()
    x = randn((n, k), 11).cuda()
    feat = torch.nn.functional.linear(x, conv.lin_src).detach().cpu().view(n, h, c)
    t_s, t_d = chain(feat, conv.att_src.detach().cpu()), chain(feat, conv.att_dst.detach().cpu())
    # of all edges that could be, those whose score lies next to zero, and some others
    edges = [torch.randint(0, n, (2, 8000), generator=torch.Generator().manual_seed(12))]
    for head in range(h):
        order = torch.sort(t_s[:, head])
        at = torch.searchsorted(order.values, -t_d[:, head].contiguous()).clamp(1, n - 1)
        for side in (0, 1):  # the source just below and just above minus the destination's score
            src = order.indices[at - side]
            small = (t_s[src, head] + t_d[:, head]).abs()
            dst = torch.sort(small).indices[:40]
            edges.append(torch.stack([src[dst], dst]))
    src, dst = torch.cat(edges, 1)
    by = torch.sort(dst, stable=True).indices
    src, dst = src[by], dst[by]
    ptr = torch.zeros(n + 1, dtype=torch.int64)
    ptr[1:] = torch.bincount(dst, minlength=n).cumsum(0)
    z = t_s[src] + t_d[dst]  # one fp32 addition, as the kernels do it
    assert int((z.abs() < 1e-7).sum()) >= 5 and int(((z > 0) & (z < 1e-6)).sum()) >= 5 and int(((z < 0) & (z > -1e-6)).sum()) >= 5

    g = randn((n, h * c), 13)
    xd = x.clone().requires_grad_()
    y = conv(xd, ptr.cuda(), src.cuda(), n, n, src.shape[0])
    names = ["x"] + [name for name, _ in conv.named_parameters()]
    got = dict(zip(names, torch.autograd.grad(y, [xd, *conv.parameters()], g.cuda())))

    # float64 from the same features, every score on the side of zero that its fp32 sum is on
    f64 = feat.double().requires_grad_()
    par = {name: p.detach().cpu().double().requires_grad_() for name, p in conv.named_parameters()}
    e = (f64 * par["att_src"]).sum(-1)[src] + (f64 * par["att_dst"]).sum(-1)[dst]
    e = torch.where(z > 0, e, 0.2 * e)
    p = torch.exp(e - e.max())
    den = torch.zeros(n, h, dtype=torch.float64).index_add(0, dst, p).clamp(min=1e-300)
    out = torch.zeros(n, h, c, dtype=torch.float64).index_add(0, dst, (p / den[dst]).unsqueeze(-1) * f64[src])
    out = out.reshape(n, h * c) + par["bias"]
    assert rel_err(y.detach().cpu(), out.detach()) < 1e-5
    gf, g_as, g_ad, gb = torch.autograd.grad(out, [f64, par["att_src"], par["att_dst"], par["bias"]], g.double())
    gf = gf.reshape(n, h * c)
    want = {"x": gf @ par["lin_src"].detach(), "lin_src": gf.t() @ x.cpu().double(), "att_src": g_as, "att_dst": g_ad, "bias": gb}
    for name in names:
        assert got[name].shape == want[name].shape and rel_err(got[name].cpu(), want[name]) < 2e-5, name
