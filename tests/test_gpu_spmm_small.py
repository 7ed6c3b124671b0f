"""cxg_spmm_csr on small graphs (one launch of clusters): every vector width and number of lanes per row, rows that lie in one tile,
cross tiles and blocks, or hold all the edges, empty rows in front, between and behind, graphs with more rows than are kept
in shared memory, against float64. The order of a sum depends on the graph only: the same bits on every run."""
import pytest
import torch

import oracle
from helpers import random_csr, randn

pytestmark = pytest.mark.gpu


def _check(ptr, idx, n_src, feat, dtype, idx_dtype=torch.int64):
    import cxgnncomp_backend as be
    n = ptr.shape[0] - 1
    assert be.SPLIT_EDGES == 0
    x, val = randn((n_src, feat), feat, dtype=dtype), randn((idx.shape[0],), feat + 1)
    deg = (ptr[1:] - ptr[:-1]).clamp(min=1).double()[:, None]
    longest = float(deg.max())
    dev = x.cuda(), ptr.cuda(), idx.to(idx_dtype).cuda(), val.cuda()
    for kw, weight in (({}, None), ({"reduce": be.CXG_MEAN}, None), ({"edge_val": dev[3]}, val)):
        before = be.kernel_launch_count()
        got = be._spmm_forward(*dev[:3], n, **kw)
        assert be.kernel_launch_count() - before == 1
        assert torch.equal(got, be._spmm_forward(*dev[:3], n, **kw))
        want = oracle.torch_spmm_index_add(x.double()[:, None], ptr, idx, n,
                                           edge_val=None if weight is None else weight.double()[:, None])[:, 0]
        if "reduce" in kw:
            want = want / deg
        # n sequential fp32 additions leave a sum, about sqrt(n) large, off by 2^-25 sqrt(n) of itself, products and the quotient
        # by another unit each; bf16 adds half of one in its eighth bit
        bound = 2 ** -25 * longest ** 0.5 + 2 ** -23 if dtype == torch.float32 else 2 ** -8
        assert (got.cpu().double() - want).norm() <= bound * want.norm()
        assert bool((got.cpu()[(ptr[1:] == ptr[:-1])] == 0).all())


@pytest.mark.parametrize("dtype,feat", [(torch.float32, f) for f in (1, 8, 9, 16, 31, 32, 33, 47, 64, 65, 66, 126, 128, 130, 256)] +
                         [(torch.bfloat16, f) for f in (1, 8, 15, 33, 34, 47, 63, 64, 128, 130, 132, 256, 260, 512)])
def test_widths(cuda, dtype, feat):
    ptr, idx = random_csr(700, 300, 9, seed=feat, hub=2500)
    _check(ptr, idx, 300, feat, dtype)


@pytest.mark.parametrize("n,deg,hub", [(1, 0, 0), (1, 3, 0), (1, 0, 40000), (5, 1, 0), (3, 0, 9000), (512, 7, 0), (513, 7, 300),
                                       (2559, 2, 0), (2560, 2, 0), (2561, 2, 50), (9000, 0, 60000), (28672, 1, 700), (20000, 0, 20000)])
@pytest.mark.parametrize("idx_dtype", [torch.int64, torch.int32])
def test_shapes(cuda, n, deg, hub, idx_dtype):
    ptr, idx = random_csr(n, 100, deg, seed=n, hub=hub, empty_frac=0.3)
    _check(ptr, idx, 100, 64, torch.float32, idx_dtype)


def test_empty_rows_at_the_ends(cuda):
    deg = torch.tensor([0] * 600 + [30, 0, 0, 500, 1] * 40 + [0] * 900)
    ptr = torch.zeros(deg.shape[0] + 1, dtype=torch.int64)
    ptr[1:] = torch.cumsum(deg, 0)
    idx = torch.randint(0, 50, (int(ptr[-1]),), generator=torch.Generator().manual_seed(1))
    _check(ptr, idx, 50, 48, torch.float32)
