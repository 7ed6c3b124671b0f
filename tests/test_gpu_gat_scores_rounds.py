"""Attention scores where a warp goes on to further nodes: one more node than all resident warps take at once and fewer, heads
of one, two and several rounds of eight vectors. Against float64; a chain of up to 256 fp32 multiply-adds, 2e-6 as in the
neighbouring tests, and the same bits wherever a node lies."""
import pytest
import torch

from helpers import randn, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,c", [(1, 32), (3, 36), (8, 32), (4, 64), (1, 256)])
def test_rounds(cuda, h, c):
    import cxgnncomp_backend as be
    full = 148 * 4 * 8 // h * 32  # nodes that the resident warps take at once
    s, d = randn((1, h, c), 2), randn((1, h, c), 3)
    x = randn((2 * full + 33, h, c), c)
    want_s, want_d = (x.double() * s.double()).sum(-1), (x.double() * d.double()).sum(-1)
    all_s, all_d = be.gat_scores(x.cuda(), s.cuda(), d.cuda(), x.shape[0])
    assert rel_err(all_s.cpu(), want_s) < 2e-6 and rel_err(all_d.cpu(), want_d) < 2e-6
    for n in (31, full - 1, full, full + 1, full + 33):
        a_s, a_d = be.gat_scores(x[:n].cuda(), s.cuda(), d.cuda(), (n + 1) // 2)
        assert torch.equal(a_s, all_s[:n]) and torch.equal(a_d, all_d[:(n + 1) // 2])
