"""The fused GAT walk at its lane layouts: head widths on both sides of the vector widths and of the rows' limits, long
chains of partials, against the op-wise formulation in float64."""
import pytest
import torch

import oracle
from helpers import random_csr, randn, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,c", [(1, 1), (2, 1), (4, 2), (1, 4), (16, 4), (2, 64), (16, 8), (8, 32), (16, 32), (8, 64),
                                     (4, 128), (1, 128), (2, 5), (8, 6), (1, 47), (4, 47), (2, 62), (8, 27), (4, 96), (4, 100),
                                     (4, 62), (1, 301), (8, 48), (16, 23)])
def test_layouts(cuda, heads, c):
    import cxgnncomp_backend as be
    n_dst, n_src = 300, 260
    ptr, idx = random_csr(n_dst, n_src, 9, seed=heads * 100 + c, hub=6000)  # more than 64 tiles of the hub row
    x, a_s, a_d = randn((n_src, heads, c), 1), randn((n_src, heads), 2) * 2, randn((n_dst, heads), 3) * 2
    xr, asr, adr = (t.double().requires_grad_(True) for t in (x, a_s, a_d))
    p = oracle.torch_edge_softmax_opwise(ptr, idx, asr, adr, idx.shape[0], 0.2)
    want = oracle.torch_spmm_index_add(xr, ptr, idx, n_dst, edge_val=p)
    train = c & (c - 1) == 0
    xg, asg, adg = (t.cuda().requires_grad_(train) for t in (x, a_s, a_d))
    with torch.set_grad_enabled(train):
        assert be.gat_fused_supported(xg)
        y, _, _ = be.gat_fused(xg, asg, adg, ptr.cuda(), idx.cuda(), n_dst, 0.2)
    assert rel_err(y.detach().cpu(), want.detach()) < 1e-5
    if not train:
        assert not be.gat_fused_supported(xg)  # gradients of such heads stay with the separate kernels
        return
    go = randn(want.shape, 4)
    want.backward(go.double())
    y.backward(go.cuda())
    assert rel_err(xg.grad.cpu(), xr.grad) < 1e-5
    assert rel_err(asg.grad.cpu(), asr.grad) < 2e-5
    assert rel_err(adg.grad.cpu(), adr.grad) < 2e-5
