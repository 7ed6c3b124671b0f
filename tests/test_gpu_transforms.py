"""torch's transforms around the operators whose hot path is a kernel call: the linear transform and the row gather follow
torch under forward-mode differentiation, vmap, tracing and fake tensors; the aggregations refuse a tangent instead of
dropping it."""
import pytest
import torch
import torch.autograd.forward_ad as fwd

from helpers import random_csr, randn, rel_err

pytestmark = pytest.mark.gpu


def test_forward_mode(cuda):
    import cxgnncomp_backend as be
    x, t, w = randn((60, 16), 1).cuda(), randn((60, 16), 2).cuda(), randn((8, 16), 3).cuda()
    rows = torch.tensor([3, 3, 50], device="cuda")
    with fwd.dual_level(), torch.no_grad():
        d = fwd.make_dual(x, t)
        got = fwd.unpack_dual(be.linear(d, w)).tangent
        assert got is not None and rel_err(got.cpu(), t.cpu().double() @ w.cpu().double().t()) < 2e-6
        assert torch.equal(fwd.unpack_dual(be.take_rows(d, rows)).tangent, t[rows])


@pytest.mark.parametrize("call", ["sum", "values", "gat", "sage"])
def test_aggregations_refuse_a_tangent(cuda, call):
    import cxgnncomp
    import cxgnncomp_backend as be
    ptr, idx = random_csr(50, 50, 5, seed=1)
    p, i = ptr.cuda(), idx.cuda()
    x, t = randn((50, 16), 1).cuda(), randn((50, 16), 2).cuda()
    val = torch.ones(idx.shape[0], device="cuda")
    att = randn((1, 4, 4), 3).cuda()
    conv = cxgnncomp.MySageConv(16, 16).cuda()
    with fwd.dual_level(), torch.no_grad():
        d = fwd.make_dual(x, t)
        with pytest.raises((RuntimeError, NotImplementedError)):
            if call == "sum":
                be.sage_sum_forward(d, p, i, 50)
            elif call == "values":
                be.sage_sum_forward_edge_value(x, p, i, fwd.make_dual(val, val), 50)
            elif call == "gat":
                be.gat_layer(d.view(50, 4, 4), att, att, None, p, i, 50, 0.2, True)
            else:
                conv(d, p, i, 50)


def test_vmap_trace_and_fake_tensors(cuda):
    import cxgnncomp
    import cxgnncomp_backend as be
    from torch._subclasses.fake_tensor import FakeTensorMode
    x, w = randn((5, 60, 16), 1).cuda(), randn((8, 16), 3).cuda()
    got = torch.func.vmap(lambda v: be.linear(v, w))(x)
    assert rel_err(got.cpu(), x.cpu().double() @ w.cpu().double().t()) < 2e-6
    layer = cxgnncomp.graph_conv.Linear(16, 8).cuda()
    with torch.no_grad():
        traced = torch.jit.trace(layer, (x[0],))
        assert rel_err(traced(x[1]).cpu(), layer(x[1]).cpu()) < 2e-6
    with FakeTensorMode(allow_non_fake_inputs=True) as mode, torch.no_grad():
        fake = mode.from_tensor(x[0])
        assert be.linear(fake, w).shape == (60, 8) and be.take_rows(fake, mode.from_tensor(torch.arange(3).cuda())).shape == (3, 16)
