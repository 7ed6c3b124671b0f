"""The register-staged tiled walk of cxg_spmm_csr at every lane layout it dispatches to: widths on both sides of the
layouts' limits, both element types, sum / mean / edge values, both index widths, tiles of one to several steps."""
import pytest
import torch

import oracle
from helpers import random_csr, randn, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,feat", [(torch.float32, f) for f in (2, 5, 8, 9, 16, 17, 33, 47, 48, 49, 65, 96, 97, 100, 129,
                                                                     193, 221, 256, 510, 512)] +
                         [(torch.bfloat16, f) for f in (3, 8, 16, 24, 47, 64, 65, 94, 100, 128, 221, 256, 258, 512)])
def test_walk_layouts(cuda, dtype, feat):
    import cxgnncomp_backend as be
    old = be.SPLIT_EDGES
    try:
        for tile, idx_dtype in ((32, torch.int64), (100, torch.int32)):
            be.SPLIT_EDGES = tile
            ptr, idx = random_csr(211, 190, 9, seed=feat + tile, hub=31 * tile // 8)
            x = randn((190, feat), feat, dtype=dtype)
            val = randn((idx.shape[0],), feat + 1)
            p, i, xg, vg = ptr.cuda(), idx.cuda().to(idx_dtype), x.cuda(), val.cuda()
            streams = feat * x.element_size() % 16 == 0 and feat * x.element_size() <= 1024
            for kw in ({}, {"mean": True}, {"edge_val": val}):
                got = be._spmm_forward(xg, p, i, 211, edge_val=vg if "edge_val" in kw else None,
                                       reduce=be.CXG_MEAN if "mean" in kw else be.CXG_SUM).cpu()
                want = oracle.spmm(ptr, idx, x, tile=tile if streams else 0, **kw)
                short = torch.ones(211, dtype=torch.bool) if streams else (ptr[1:] - ptr[:-1]) <= tile
                assert torch.equal(got[short], want[short]), (tile, kw.keys())
                assert rel_err(got.float(), want.float()) < (1e-5 if dtype == torch.float32 else 2 ** -7)
    finally:
        be.SPLIT_EDGES = old
