"""Sampling a batch where the nodes per block change: frontiers of one block's share and one node more or less, and on both
sides of the sizes from which blocks take more nodes, for 8, 16 and 32 lanes a node. Bit for bit what the hop-by-hop entry
points give."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fanout,seeds", [(3, 31), (3, 33), (3, 65567), (3, 65568), (12, 15), (12, 16), (12, 17), (12, 32783), (12, 32784),
                                          (20, 7), (20, 8), (20, 9), (20, 16391), (20, 16392), (2, 262207), (2, 262208)])
def test_blocks(cuda, fanout, seeds, monkeypatch):
    import cxgnncomp
    import cxgnncomp_backend as be
    from cxgnncomp import synthetic
    n = max(2 * seeds, 5000) if seeds < 100000 else seeds + 1000
    ptr, idx = synthetic.powerlaw_graph(n, 4 * n, seed=fanout)
    s = torch.randperm(n, generator=torch.Generator().manual_seed(seeds))[:seeds].cuda()
    sampler = cxgnncomp.NeighborSampler(ptr.cuda(), idx.cuda(), [fanout, 2])
    got = [sampler.sample(s, seed=k) for k in (5, 6)]
    assert bool((sampler.local_of == -1).all()) and not bool(sampler._marks.any())
    monkeypatch.setattr(be, "sample_batch_fits", lambda *a: False)
    want = [sampler.sample(s, seed=k) for k in (5, 6)]
    for g, w in zip(got, want):
        assert g[3] == w[3] and g[4] == w[4]
        for a, b in zip(g[:3], w[:3]):
            assert torch.equal(a, b)
