"""The RGCN layer's training path over the distinct (relation, source) pairs: output and gradients against float64, at
widths on both sides of the kernels' tiles, relations without edges, sources without pairs, rows without edges."""
import pytest
import torch

from helpers import random_csr, randn, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-6), (torch.bfloat16, 2e-2)])
@pytest.mark.parametrize("k,o,R,n", [(128, 64, 8, 900), (16, 16, 2, 50), (48, 112, 12, 400), (96, 128, 1, 130), (32, 64, 5, 3000)])
def test_layer(cuda, dtype, tol, k, o, R, n):
    import cxgnncomp
    import cxgnncomp_backend as be
    ptr, idx = random_csr(n, n, 7, seed=k + o, hub=1500)
    rel = torch.randint(0, max(1, R - 1), (idx.shape[0],), generator=torch.Generator().manual_seed(n))  # the last one is empty
    conv = cxgnncomp.MyRGCNConv(k, o, R).cuda().to(dtype)
    x, go = randn((n, k), 1).to(dtype), randn((n, o), 2).to(dtype)
    xg = x.cuda().requires_grad_(True)
    p, i, rg = ptr.cuda(), idx.cuda(), rel.cuda()
    assert be.relation_pairs_supported(xg, conv.linear)
    y = conv(xg, p, i, rg, n)
    y.backward(go.cuda())
    xr, wr = x.double().requires_grad_(True), conv.linear.detach().cpu().double().requires_grad_(True)
    dst = torch.repeat_interleave(torch.arange(n), ptr[1:] - ptr[:-1])
    want = torch.zeros(n, o, dtype=torch.float64)
    for r in range(R):
        e = (rel == r).nonzero().squeeze(1)
        want = want.index_add(0, dst[e], xr[idx[e]] @ wr[r])
    want = want / (ptr[1:] - ptr[:-1]).clamp(min=1).double()[:, None]
    want.backward(go.double())
    assert rel_err(y.detach().cpu(), want.detach()) < tol
    assert rel_err(xg.grad.cpu(), xr.grad) < tol and rel_err(conv.linear.grad.cpu(), wr.grad) < tol
    first = xg.grad.clone()
    xg.grad = None
    conv(xg, p[:], i[:], rg[:], n).backward(go.cuda())  # other tensor objects of the same graph, same bits
    assert torch.equal(xg.grad, first)
