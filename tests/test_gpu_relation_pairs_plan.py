"""The distinct (relation, source) pairs of a graph against their definition on the host: numbers of sources on both sides of
a word and of a block of words, relations without edges, many relations, both index widths; edges outside the ranges."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def definition(idx, rel, n, R):
    pairs = torch.unique(rel.long() * n + idx.long())
    pr, ps = pairs // n, pairs % n
    pos_rel, pos_src, where = [], [], {}
    for r in range(R):
        src = ps[pr == r].tolist()
        padded = (len(src) + 127) // 128 * 128
        for j, s in enumerate(src):
            where[(r, s)] = len(pos_src) + j
        pos_src += src + [-1] * (padded - len(src))
        pos_rel += [r] * padded
    lists = [[where[(r, s)] for r in range(R) if (r, s) in where] for s in range(n)]
    src_ptr = torch.tensor([0] + [len(x) for x in lists]).cumsum(0)
    return (pos_rel, pos_src, list(range(len(pos_src))), src_ptr.tolist(), [p for x in lists for p in x],
            [where[(int(r), int(s))] for r, s in zip(rel, idx)])


@pytest.mark.parametrize("n,R,nnz", [(1, 1, 3), (31, 2, 40), (32, 3, 500), (33, 1, 20), (500, 8, 4000), (4096, 3, 9000),
                                     (8192, 2, 20000), (8193, 5, 30000), (20000, 4, 300), (40, 300, 5000)])
@pytest.mark.parametrize("idx_dtype,rel_dtype", [(torch.int64, torch.int64), (torch.int32, torch.int64), (torch.int64, torch.int32),
                                                 (torch.int32, torch.uint8)])
def test_plan(cuda, n, R, nnz, idx_dtype, rel_dtype):
    import cxgnncomp_backend as be
    if rel_dtype == torch.uint8 and R > 255:
        pytest.skip("relation ids do not fit")
    gen = torch.Generator().manual_seed(n + R)
    # a few sources have most of the edges, and the last relation of several has none
    idx = (torch.rand(nnz, generator=gen) ** 3 * n).long().clamp(max=n - 1)
    rel = torch.randint(0, max(1, R - 1), (nnz,), generator=gen)
    got = be.RelationPairs(idx.to(idx_dtype).cuda(), rel.to(rel_dtype).cuda(), n, R)
    want = definition(idx, rel, n, R)
    for a, b in zip((got.rel, got.src, got.pos, got.src_ptr, got.src_idx, got.idx), want):
        assert a.tolist() == b
    assert got.num_pos == len(want[0])


def test_edges_outside(cuda):
    import cxgnncomp_backend as be
    idx, rel = torch.tensor([0, 4, 2]), torch.tensor([0, 1, 1])
    for i, r in ((idx + 1, rel), (idx - 1, rel), (idx, rel + 1), (idx, rel - 1)):
        with pytest.raises(RuntimeError, match="edge types must lie in"):
            be.RelationPairs(i.cuda(), r.cuda(), 5, 2)
    assert be.RelationPairs(idx.cuda(), rel.cuda(), 5, 2).num_pos == 256


def test_kept_plans(cuda, monkeypatch):
    """The last eight graphs, fewer beyond the byte limit, none after forget_graphs; a plan serves another stream."""
    import cxgnncomp_backend as be
    be.forget_graphs()
    gen = torch.Generator().manual_seed(9)
    graphs = [(torch.randint(0, 300, (5000,), generator=gen).cuda(), torch.randint(0, 4, (5000,), generator=gen).cuda()) for _ in range(10)]
    plans = [be.relation_pairs(i, r, 300, 4) for i, r in graphs]
    assert len(be._pair_cache) == 8 and be.relation_pairs(*graphs[9], 300, 4) is plans[9]
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        assert be.relation_pairs(*graphs[9], 300, 4) is plans[9]
        fresh = be.relation_pairs(*graphs[0], 300, 4)
    torch.cuda.current_stream().wait_stream(side)
    assert fresh is not plans[0] and all(torch.equal(a, b) for a, b in zip(fresh.tensors(), plans[0].tensors()))
    monkeypatch.setattr(be, "_PAIR_CACHE_BYTES", 1)
    be.relation_pairs(*graphs[1], 300, 4)
    assert len(be._pair_cache) == 1
    be.forget_graphs()
    assert not be._pair_cache and len(be._TRANSPOSE_CACHE) == 0
