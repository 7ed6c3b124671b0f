"""The register-staged walk when there are more tiles than are walked at once (tiles handed out one by one), and its chains of
partial sums over many tiles, for widths that are whole vectors and widths that are not: bit for bit against the oracle."""
import pytest
import torch

import oracle
from helpers import random_csr, randn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,feat", [(torch.float32, 4), (torch.float32, 64), (torch.float32, 128), (torch.bfloat16, 24),
                                        (torch.float32, 9), (torch.float32, 47), (torch.bfloat16, 33)])
@pytest.mark.parametrize("kw", [{}, {"mean": True}, {"edge_val": True}], ids=["sum", "mean", "value"])
def test_more_tiles_than_groups(cuda, dtype, feat, kw):
    import cxgnncomp_backend as be
    n, tile = 5000, 8
    ptr, idx = random_csr(n, 900, 40, seed=feat, hub=9000)
    assert idx.shape[0] > tile * 148 * 8 * 16  # the most groups that are resident
    x, val = randn((900, feat), feat, dtype=dtype), randn((idx.shape[0],), feat + 1)
    streams = feat * x.element_size() % 16 == 0
    oracle_kw = dict(kw, edge_val=val) if "edge_val" in kw else kw
    old = be.SPLIT_EDGES
    try:
        be.SPLIT_EDGES = tile
        got = be._spmm_forward(x.cuda(), ptr.cuda(), idx.cuda(), n, edge_val=val.cuda() if "edge_val" in kw else None,
                               reduce=be.CXG_MEAN if "mean" in kw else be.CXG_SUM).cpu()
    finally:
        be.SPLIT_EDGES = old
    want = oracle.spmm(ptr, idx, x, tile=tile if streams else 0, **oracle_kw)
    short = torch.ones(n, dtype=torch.bool) if streams else (ptr[1:] - ptr[:-1]) <= tile
    assert torch.equal(got[short], want[short])
    # Rows that are cut are summed in another order than the oracle's. n sequential fp32 additions of terms like these leave the
    # sum, about sqrt(n) large, off by a random walk of n steps of half a unit in its last place each, at most 2^-25 sqrt(n):
    # relative to the result 2^-25 sqrt(n) on either side, n = 9,000 at most. bf16 adds one rounding.
    err = (got.double() - want.double()).norm() / want.double().norm()
    assert err < (2 * 2 ** -25 * 9000 ** 0.5 if dtype == torch.float32 else 2 ** -8)
