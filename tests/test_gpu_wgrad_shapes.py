"""The typed weight gradient at widths on both sides of its 128-byte spans, against float64: columns behind K and N, tiles
narrower than the 128 columns the tensor core reads, one and several relations."""
import pytest
import torch

from helpers import randn, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("k,n", [(8, 16), (16, 16), (32, 16), (40, 48), (64, 32), (72, 112), (96, 64), (112, 128), (128, 16),
                                 (128, 48), (128, 128)])
def test_widths(cuda, dtype, k, n):
    import cxgnncomp_backend as be
    R, blocks = 5, [3, 0, 1, 17, 2]  # 128-position blocks per relation
    m = 128 * sum(blocks)
    rel = torch.repeat_interleave(torch.arange(R), torch.tensor(blocks) * 128)
    x, g = randn((m, k), k).to(dtype), randn((m, n), n + 1).to(dtype)
    idx = torch.randperm(m, generator=torch.Generator().manual_seed(k * n))
    idx[torch.rand(m, generator=torch.Generator().manual_seed(n)) < 0.2] = -1  # padding
    assert be.typed_wgrad_supported(x.cuda(), g.cuda())
    got = be.typed_wgrad(x.cuda(), g.cuda(), rel.cuda(), R, idx=idx.cuda(), check_status=True).cpu()
    for r in range(R):
        rows = idx[(rel == r) & (idx >= 0)]
        want = x[rows].double().t() @ g[rows].double()
        assert rel_err(got[r], want) < 2e-6 if rows.numel() else not bool(got[r].any())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("k,n", [(8, 16), (32, 48), (40, 48), (72, 112), (96, 64), (64, 256), (16, 256)])
def test_every_stage(cuda, dtype, k, n):
    """As many tiles as every block of the kernel needs to go through all stages of its ring several times: narrow operands
    are read beyond their own columns, behind the last stage into room of their own."""
    import cxgnncomp_backend as be
    R, m = 3, 128 * 148 * 12
    rel = (torch.arange(m // 128) * R // (m // 128)).repeat_interleave(128)
    x, g = randn((m, k), k).to(dtype), randn((m, n), n + 1).to(dtype)
    got = be.typed_wgrad(x.cuda(), g.cuda(), rel.cuda(), R, check_status=True).cpu()
    for r in range(R):
        rows = rel == r
        assert rel_err(got[r], x[rows].double().t() @ g[rows].double()) < 4e-6
