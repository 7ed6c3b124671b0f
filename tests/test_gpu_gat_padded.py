"""GAT layers in inference whose heads are not whole 16-byte vectors: transformed with padded heads (gat_layer_padded), against the
layer's op-by-op form in float64."""
import pytest
import torch

from helpers import random_csr, randn, rel_err

pytestmark = pytest.mark.gpu


def _exact(conv, x, ptr, idx, n):
    h, c = conv.heads, conv.out_channels
    f = (x.double() @ conv.lin_src.double().t()).view(-1, h, c)
    a_s, a_d = (f * conv.att_src.double()).sum(-1), (f[:n] * conv.att_dst.double()).sum(-1)
    dst = torch.repeat_interleave(torch.arange(n, device=x.device), ptr[1:n + 1] - ptr[:n])
    t = torch.nn.functional.leaky_relu(a_s[idx] + a_d[dst], conv.negative_slope)
    top = torch.full((n, h), -torch.inf, dtype=torch.float64, device=x.device).scatter_reduce(0, dst[:, None].expand(-1, h), t, "amax")
    p = torch.exp(t - top[dst])
    p = p / torch.zeros(n, h, dtype=torch.float64, device=x.device).index_add_(0, dst, p)[dst]
    y = torch.zeros(n, h, c, dtype=torch.float64, device=x.device).index_add_(0, dst, p[:, :, None] * f[idx])
    y = y.reshape(n, h * c) if conv.concat else y.mean(1)
    return y if conv.bias is None else y + conv.bias.double()


@pytest.mark.parametrize("heads,c", [(2, 9), (2, 13), (4, 47), (4, 11), (8, 17), (8, 62), (2, 255)])
@pytest.mark.parametrize("concat,bias", [(True, True), (False, True), (False, False)])
def test_layer(cuda, heads, c, concat, bias):
    import cxgnncomp
    import cxgnncomp_backend as be
    n_dst, n_src, k = 230, 260, 36
    ptr, idx = (t.cuda() for t in random_csr(n_dst, n_src, 9, seed=heads * 100 + c, hub=3000))
    torch.manual_seed(c)
    conv = cxgnncomp.MyGATConv(k, c, heads=heads, concat=concat, bias=bias).cuda()
    if bias:
        conv.bias.data.normal_()
    x = randn((n_src, k), 5).cuda()
    with torch.no_grad():
        assert be.gat_layer_padded(x, conv.lin_src, conv.att_src, conv.att_dst, conv.bias, ptr, idx, n_dst, heads, 0.2, concat) is not None
        y = conv(x, ptr, idx, n_dst, n_src, idx.shape[0])
        assert y.shape == (n_dst, heads * c if concat else c)
        assert rel_err(y, _exact(conv, x, ptr, idx, n_dst)) < 1e-5


def test_not_covered(cuda):
    import cxgnncomp
    import cxgnncomp_backend as be
    ptr, idx = (t.cuda() for t in random_csr(50, 60, 5, seed=1))
    x = randn((60, 16), 5).cuda()

    def padded(c, x=x):
        conv = cxgnncomp.MyGATConv(16, c, heads=2).cuda()
        return be.gat_layer_padded(x, conv.lin_src, conv.att_src, conv.att_dst, conv.bias, ptr, idx, 50, 2, 0.2, False)

    assert padded(9) is None  # gradients are recorded
    with torch.no_grad():
        assert padded(9) is not None
        assert padded(7) is None and padded(12) is None and padded(257) is None
        assert padded(9, x.double()) is None and padded(9, randn((60, 32), 5).cuda()[:, ::2]) is None
        with torch.autocast("cuda", dtype=torch.bfloat16):
            assert padded(9) is None
