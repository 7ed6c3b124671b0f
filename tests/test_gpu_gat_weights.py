"""The fused GAT forward by way of weights (cxg_gat_fused_forward, all widths but vectors across heads, narrow rows of whole
vectors from 128 MB of gathered rows on): rows of one edge to thousands, on both sides of what a lane and a warp keep in registers, rows that cross tiles, empty rows, every vector width
and number of heads, against float64."""
import pytest
import torch

import oracle
from helpers import randn, rel_err

pytestmark = pytest.mark.gpu


def _graph(degrees, n_src, seed):
    g = torch.Generator().manual_seed(seed)
    deg = torch.tensor(degrees)[torch.randperm(len(degrees), generator=g)]
    ptr = torch.zeros(len(degrees) + 1, dtype=torch.int64)
    ptr[1:] = torch.cumsum(deg, 0)
    return ptr, torch.randint(0, n_src, (int(ptr[-1]),), generator=g)


@pytest.mark.parametrize("heads,c", [(1, 47), (1, 50), (1, 256), (2, 33), (2, 15), (2, 66), (4, 64), (4, 33), (8, 20), (8, 64),
                                     (2, 10), (4, 6), (8, 2), (4, 5), (8, 7)])
@pytest.mark.parametrize("idx_dtype", [torch.int64, torch.int32])
def test_forward(cuda, heads, c, idx_dtype):
    import cxgnncomp_backend as be
    n_src = 700
    step = 32 // heads
    lengths = [0, 1, 2, 7, 8, 9, 15, 16, 17, 8 * step - 1, 8 * step, 8 * step + 1, 300, 1500]
    degrees = [lengths[i % len(lengths)] for i in range(160)] + [0, 0, 4000] + [5] * 200 + [0] * 3
    ptr, idx = _graph(degrees, n_src, heads * 100 + c)
    n = len(degrees)
    x, a_s, a_d = randn((n_src, heads, c), 1), randn((n_src, heads), 2) * 2, randn((n, heads), 3) * 2
    p = oracle.torch_edge_softmax_opwise(ptr, idx, a_s.double(), a_d.double(), idx.shape[0], 0.2)
    want = oracle.torch_spmm_index_add(x.double(), ptr, idx, n, edge_val=p)
    with torch.no_grad():
        y, top, total = (t.cpu() for t in be.gat_fused(x.cuda(), a_s.cuda(), a_d.cuda(), ptr.cuda(), idx.to(idx_dtype).cuda(), n, 0.2))
    assert rel_err(y, want) < 1e-5
    deg = ptr[1:] - ptr[:-1]
    has = deg > 0
    t = torch.nn.functional.leaky_relu(a_s.double()[idx] + torch.repeat_interleave(a_d.double(), deg, dim=0), 0.2)
    mx = torch.segment_reduce(t, "max", lengths=deg, unsafe=True)
    sm = torch.segment_reduce(torch.exp(t - torch.repeat_interleave(mx, deg, dim=0)), "sum", lengths=deg, unsafe=True)
    assert torch.allclose(top.double()[has], mx[has], atol=1e-6, rtol=1e-6)
    assert torch.allclose(total.double()[has], sm[has], rtol=1e-5)
    assert bool((total[~has] == 0).all()) and bool((y[~has] == 0).all())


def test_large_scores(cuda):
    """Scores whose exponentials overflow without the maximum taken out, and rows in which one edge has all the weight."""
    import cxgnncomp_backend as be
    ptr, idx = _graph([3, 40, 0, 900, 1, 12] * 20, 300, 5)
    n = ptr.shape[0] - 1
    x, a_s, a_d = randn((300, 4, 64), 1), randn((300, 4), 2) * 300, randn((n, 4), 3) * 300
    p = oracle.torch_edge_softmax_opwise(ptr, idx, a_s.double(), a_d.double(), idx.shape[0], 0.2)
    want = oracle.torch_spmm_index_add(x.double(), ptr, idx, n, edge_val=p)
    with torch.no_grad():
        y = be.gat_fused(x.cuda(), a_s.cuda(), a_d.cuda(), ptr.cuda(), idx.cuda(), n, 0.2)[0]
    # a score near 1000 is rounded by 2^-15 and its weight by as much, in the row's other terms too
    assert rel_err(y.cpu(), want) < 4 * 2 ** -15


def test_no_edges(cuda):
    import cxgnncomp_backend as be
    ptr, idx = torch.zeros(101, dtype=torch.int64).cuda(), torch.empty(0, dtype=torch.int64).cuda()
    y, _, total = be.gat_fused(randn((50, 4, 64), 1).cuda(), randn((50, 4), 2).cuda(), randn((100, 4), 3).cuda(), ptr, idx, 100, 0.2)
    assert bool((y == 0).all()) and bool((total == 0).all())


@pytest.mark.parametrize("heads,c", [(2, 16), (2, 32), (4, 8), (4, 16), (8, 4), (8, 8), (8, 12)])
def test_last_tile_of_one_edge(cuda, heads, c):
    """The fewest edges from which these widths go by weights, 8 and 16 lanes per tile, and one more than whole tiles."""
    import ctypes
    import cxgnncomp_backend as be
    room = be._lib.cxg_gat_fused_weights_room
    room.argtypes = [ctypes.c_int64, ctypes.c_int64, ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_size_t)]
    tile, size = ctypes.c_int(0), ctypes.c_size_t(0)
    n_src, edges = 5000, (128 << 20) // (heads * c * 4) + 1
    assert room(1, edges, heads, c, ctypes.byref(tile), ctypes.byref(size)) == 0 and tile.value > 0
    edges += -(edges - 1) % tile.value
    deg = torch.randint(0, 60, (edges // 30 + 2000,), generator=torch.Generator().manual_seed(c))
    ptr = torch.zeros(deg.numel() + 1, dtype=torch.int64)
    ptr[1:] = torch.cumsum(deg, 0).clamp(max=edges)
    assert int(ptr[-1]) == edges and edges % tile.value == 1
    idx = torch.randint(0, n_src, (edges,), generator=torch.Generator().manual_seed(heads))
    n = deg.numel()
    x, a_s, a_d = randn((n_src, heads, c), 1), randn((n_src, heads), 2), randn((n, heads), 3)
    p = oracle.torch_edge_softmax_opwise(ptr.cuda(), idx.cuda(), a_s.double().cuda(), a_d.double().cuda(), edges, 0.2)
    want = oracle.torch_spmm_index_add(x.double().cuda(), ptr.cuda(), idx.cuda(), n, edge_val=p)
    with torch.no_grad():
        y = be.gat_fused(x.cuda(), a_s.cuda(), a_d.cuda(), ptr.cuda(), idx.cuda(), n, 0.2)[0]
    assert rel_err(y, want) < 1e-5
