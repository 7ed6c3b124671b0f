"""Sums and means that are added to the output on the tiled walk, at its lane layouts: the oracle's order bit for bit (rows cut
by tiles included), rows without edges left as they are, the grid that leaves room on the SMs, a graph without edges."""
import pytest
import torch

import oracle
from helpers import random_csr, randn, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,feat", [(torch.float32, f) for f in (1, 8, 9, 33, 47, 64, 100, 128, 193, 256, 512)] +
                         [(torch.bfloat16, f) for f in (3, 16, 24, 47, 64, 94, 128, 221, 256, 512)])
@pytest.mark.parametrize("mean", [False, True])
def test_added_to(cuda, dtype, feat, mean):
    import cxgnncomp_backend as be
    old = be.SPLIT_EDGES
    try:
        for tile, idx_dtype in ((32, torch.int64), (100, torch.int32)):
            be.SPLIT_EDGES = tile
            ptr, idx = random_csr(211, 190, 9, seed=feat + tile, hub=70 * tile)
            x, base = randn((190, feat), feat, dtype=dtype), randn((211, feat), feat + 1, dtype=dtype)
            p, i, xg = ptr.cuda(), idx.cuda().to(idx_dtype), x.cuda()
            streams = feat * x.element_size() % 16 == 0 and feat * x.element_size() <= 1024
            want = oracle.spmm(ptr, idx, x, tile=tile if streams else 0, mean=mean, out=base)
            deg = ptr[1:] - ptr[:-1]
            exact = torch.ones(211, dtype=torch.bool) if streams else deg <= tile
            for share in (False, True):
                got = base.cuda()
                be.spmm_into(got, p, i, xg, 211, reduce="mean" if mean else "sum", accumulate=True, share_sms=share)
                got = got.cpu()
                assert torch.equal(got[exact], want[exact]) and torch.equal(got[deg == 0], base[deg == 0])
                assert rel_err(got.float(), want.float()) < (1e-5 if dtype == torch.float32 else 2 ** -7)
            rel = torch.randint(0, 2, (idx.shape[0],), generator=torch.Generator().manual_seed(1), dtype=torch.int32)
            got = base.cuda()
            be._spmm_forward(xg, p, i % 95, 211, out=got, accumulate=True, edge_rel=rel.cuda(), rel_stride=95)
            want = oracle.spmm(ptr, idx % 95, x, tile=tile if streams else 0, edge_rel=rel, rel_stride=95, out=base)
            assert torch.equal(got.cpu()[exact], want[exact])
        got = base.cuda()
        be.spmm_into(got, torch.zeros(212, dtype=torch.int64, device="cuda"), p.new_zeros(0), xg, 211, accumulate=True)
        assert torch.equal(got.cpu(), base)
    finally:
        be.SPLIT_EDGES = old
