"""More source rows than 32 bits can number (one bf16 column of them is 8.6 GB)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_rows_behind_two_to_the_32(cuda):
    import cxgnncomp_backend as be
    n = (1 << 32) + 8
    if torch.cuda.get_device_properties(0).total_memory < 40 << 30:
        pytest.skip("needs 9 GB")
    x = torch.zeros(n, 1, dtype=torch.bfloat16, device="cuda")
    x[5], x[(1 << 32) + 5], x[(1 << 32) - 1] = 7, 3, 2
    ptr = torch.tensor([0, 1, 2, 4, 4], device="cuda")
    idx = torch.tensor([(1 << 32) + 5, 5, (1 << 32) - 1, (1 << 32) + 5], device="cuda")
    assert be.sage_sum_forward(x, ptr, idx, 4).flatten().tolist() == [3, 7, 5, 0]
    y = torch.ones(4, 1, dtype=torch.bfloat16, device="cuda")
    be.spmm_into(y, ptr, idx, x, 4, accumulate=True)
    assert y.flatten().tolist() == [4, 8, 6, 1]
