"""The typed matmul on the tensor cores at widths that give every span of its swizzled layout (128, 64 and 32 bytes) and
K-blocks of one and several spans, against float64: gathered rows, padding, and all relations at once."""
import pytest
import torch

from helpers import randn, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["compensated", "tf32", "bf16"])
@pytest.mark.parametrize("k,n", [(16, 16), (32, 48), (48, 64), (64, 16), (80, 32), (96, 128), (112, 96), (128, 64), (128, 208),
                                 (192, 128), (208, 64), (256, 96), (432, 256), (1744, 16)])
def test_spans(cuda, mode, k, n):
    import cxgnncomp_backend as be
    dtype, tol = {"compensated": (torch.float32, 2e-6), "tf32": (torch.float32, 2e-3), "bf16": (torch.bfloat16, 5e-3)}[mode]
    R, blocks = 4, [2, 0, 1, 3]  # 128-position blocks per relation
    tol *= max(1.0, k / 512)  # the tensor core cuts its sum at every step of K
    m, rows = 128 * sum(blocks), 500
    if n * k * (2 if mode == "bf16" else 4) + 128 * 32 > 226 * 1024:
        pytest.skip("W does not fit in shared memory")
    rel = torch.repeat_interleave(torch.arange(R), torch.tensor(blocks) * 128)
    x, w = randn((rows, k), k).to(dtype), randn((R, k, n), n + 1).to(dtype)
    idx = torch.randint(0, rows, (m,), generator=torch.Generator().manual_seed(k * n))
    idx[torch.rand(m, generator=torch.Generator().manual_seed(n)) < 0.2] = -1  # padding
    got = be.typed_matmul_raw(x.cuda(), w.cuda(), rel.cuda(), m, rows, src_idx=idx.cuda(), seq_output=True,
                              allow_tf32=mode == "tf32").cpu()
    for r in range(R):
        sel = (rel == r) & (idx >= 0)
        if sel.any():
            assert rel_err(got[sel], x[idx[sel]].double() @ w[r].double()) < tol
    if mode != "tf32" and be.typed_matmul_all_relations_supported(x.cuda(), w.cuda()):
        got = be.typed_matmul_all_relations(x.cuda(), w.cuda()).cpu()
        assert rel_err(got.view(R, rows, n), torch.einsum("mk,rkn->rmn", x.double(), w.double())) < tol
