"""The typed weight gradient where a block adds several accumulators to one relation's sum: ranges of more than 4,096
positions, relations that change inside and between them, widths that give the two groups of epilogue warps unequal shares.
Against float64. The tensor core cuts its sum at every instruction, by at most 2^-23 of it: 256 instructions of 16 bf16
products in an accumulator, whose sum grows from nothing, are short by at most 256 * 2^-23 / 2 = 1.5e-5 of the result; 32
instructions of the compensated mode by 2e-6, and as much for the terms it leaves out."""
import pytest
import torch

from helpers import randn, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,blocks,bound", [(torch.bfloat16, 70, 1.5e-5), (torch.float32, 9, 4e-6)])
@pytest.mark.parametrize("k,n", [(16, 48), (72, 80), (128, 16), (104, 144)])
def test_chunks(cuda, dtype, blocks, bound, k, n):
    import cxgnncomp_backend as be
    m = 128 * 148 * blocks
    cut = 128 * (m // 300)  # somewhere inside a block's range
    rel = torch.zeros(m, dtype=torch.int64)
    rel[cut:] = 1
    rel[-128:] = 2
    x, g = randn((m, k), k).to(dtype), randn((m, n), n + 1).to(dtype)
    got = be.typed_wgrad(x.cuda(), g.cuda(), rel.cuda(), 3, check_status=True).cpu()
    for r, rows in enumerate((slice(0, cut), slice(cut, m - 128), slice(m - 128, m))):
        assert rel_err(got[r], x[rows].double().t() @ g[rows].double()) < bound
