"""Aggregation from rows that the call has copied to whole lines (cxg_spmm_csr_rows): the bits of the call that reads x as it is,
for the widths, types and alignments that take the copy and around its limits."""
import ctypes

import pytest
import torch

from helpers import random_csr, randn

pytestmark = pytest.mark.gpu


def _sizes(be, desc, n_src):
    fn = be._lib.cxg_spmm_csr_rows_size
    fn.argtypes, fn.restype = [ctypes.POINTER(be.SpmmDesc), ctypes.c_int64, ctypes.POINTER(ctypes.c_size_t)], ctypes.c_int
    need = ctypes.c_size_t(0)
    assert fn(ctypes.byref(desc), n_src, ctypes.byref(need)) == 0
    return need.value


def _plain(be, x, ptr, idx, n, val, reduce):
    """The call without scratch for the rows, and the bytes that the other one would copy them to."""
    y = torch.empty((n, x.shape[1]), dtype=x.dtype, device="cuda")
    desc = be._make_desc(ptr, idx, x, y, n, feat=x.shape[1], edge_val=val, reduce=reduce)
    need = ctypes.c_size_t(0)
    assert be._spmm_ws(n, idx.shape[0], x.shape[1], 1, be.SPLIT_EDGES, ctypes.byref(need)) == 0
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    be._check(be._spmm_fwd(ctypes.byref(desc), be._p(ws), need.value, be._stream()), "cxg_spmm_csr")
    torch.cuda.synchronize()
    return y, _sizes(be, desc, x.shape[0])


@pytest.mark.parametrize("dtype,feat,copied", [
    (torch.float32, 16, False), (torch.float32, 17, True), (torch.float32, 31, True), (torch.float32, 32, False),
    (torch.float32, 33, True), (torch.float32, 46, True), (torch.float32, 47, True), (torch.float32, 65, True),
    (torch.float32, 97, True), (torch.float32, 127, True), (torch.float32, 129, True), (torch.float32, 100, False),
    (torch.float32, 255, True), (torch.bfloat16, 33, True), (torch.bfloat16, 50, True), (torch.bfloat16, 63, True),
    (torch.bfloat16, 65, True), (torch.bfloat16, 101, True), (torch.bfloat16, 104, False), (torch.bfloat16, 255, True)])
@pytest.mark.parametrize("idx_dtype", [torch.int64, torch.int32])
def test_same_bits_as_without_the_copy(cuda, dtype, feat, copied, idx_dtype):
    import cxgnncomp_backend as be
    n, n_src = 3000, 2500
    degree = (44 << 20) // (feat * (4 if dtype == torch.float32 else 2)) // n * 10 // 9 + 16
    ptr, idx = random_csr(n, n_src, degree, seed=feat, hub=5000)
    ptr, idx, x = ptr.cuda(), idx.to(idx_dtype).cuda(), randn((n_src, feat), feat, dtype=dtype).cuda()
    val = randn((idx.shape[0],), feat + 1).cuda()
    old = be.SPLIT_EDGES
    try:
        be.SPLIT_EDGES = 96
        for v, reduce in ((None, be.CXG_SUM), (None, be.CXG_MEAN), (val, be.CXG_SUM)):
            want, rows = _plain(be, x, ptr, idx, n, v, reduce)
            assert (rows > 0) == copied
            got = be._spmm_forward(x, ptr, idx, n, edge_val=v, reduce=reduce)
            assert torch.equal(got, want)
    finally:
        be.SPLIT_EDGES = old


def test_rows_that_start_between_vectors(cuda):
    """Rows of whole vectors whose first one is not: the copy aligns them."""
    import cxgnncomp_backend as be
    n, n_src, feat = 2000, 1500, 64
    ptr, idx = random_csr(n, n_src, 120, seed=3, hub=3000)
    x = randn((n_src * feat + 1,), 4).cuda()[1:].view(n_src, feat)
    assert x.data_ptr() % 16 == 4
    want, rows = _plain(be, x, ptr.cuda(), idx.cuda(), n, None, be.CXG_SUM)
    assert rows == n_src * 256
    old = be.SPLIT_EDGES
    got = be._spmm_forward(x, ptr.cuda(), idx.cuda(), n)
    ref = be._spmm_forward(x.clone(), ptr.cuda(), idx.cuda(), n)
    assert be.SPLIT_EDGES == old
    # other tiles, other order: 2^-25 sqrt(3000) on either side
    for other in (want, ref):
        assert (got.double() - other.double()).norm() < 2 * 2 ** -25 * 3000 ** 0.5 * other.double().norm()


def test_few_edges_read_x_as_it_is(cuda):
    import cxgnncomp_backend as be
    ptr, idx = random_csr(500, 20000, 400, seed=1)
    x = randn((20000, 47), 1).cuda()
    assert _plain(be, x, ptr.cuda(), idx.cuda(), 500, None, be.CXG_SUM)[1] == 0
