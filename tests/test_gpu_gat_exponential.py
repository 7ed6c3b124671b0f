"""The exponential of the fused GAT walk against its stated bound, (1.5 |x| + 4) * 2^-24 of the result and zero below 2^-126:
rows of two edges whose scores are x apart and whose features are 0 and 1, in both orders (the walk rescales in one of them)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,c", [(1, 4), (4, 32), (2, 15), (4, 47), (1, 128), (2, 256)])
def test_two_edges(cuda, h, c):
    import cxgnncomp_backend as be
    n = 4000
    # multiples of 2^-16 below 100: the scores and their differences are exact
    x = torch.randint(0, 87 << 16, (n,), generator=torch.Generator().manual_seed(c)).double() / 65536
    x[:4] = torch.tensor([0, 2 ** -16, 87.5, 99.0])
    score = torch.cat([torch.tensor([100.0]).double(), 100 - x]).float()
    feat = torch.ones(n + 1, h, c)
    feat[0] = 0
    k = torch.arange(1, n + 1)
    ptr = torch.arange(0, 4 * n + 1, 2)
    idx = torch.stack([torch.zeros(n, dtype=torch.int64), k, k, torch.zeros(n, dtype=torch.int64)], 1).flatten()
    a_src = score[:, None].expand(n + 1, h).contiguous()
    with torch.no_grad():
        y, top, total = be.gat_fused(feat.cuda(), a_src.cuda(), torch.zeros(2 * n, h, device="cuda"), ptr.cuda(), idx.cuda(),
                                     2 * n, 0.2)
    e = torch.exp(-x)
    want = (e / (1 + e)).repeat_interleave(2)[:, None, None]
    err = ((y.cpu().double() - want) / want).abs()
    # and the sum, its reciprocal and the product with it: 2^-24 each and as much again for an approximate reciprocal
    bound = (1.5 * x + 4 + 4).repeat_interleave(2)[:, None, None] * 2.0 ** -24
    kept = (e >= 2.0 ** -126).repeat_interleave(2)
    assert bool((err <= bound)[kept].all()), float((err / bound)[kept].max())
    assert not bool(y.cpu()[~kept].any()) and bool((top == 100).all())
    assert float((total.cpu().double() - (1 + e).repeat_interleave(2)[:, None]).abs().max()) < 3e-7
