"""Sampling a batch in one call against the hop-by-hop entry points: same nodes, rows, neighbours and sizes, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fanouts", [[15, 10, 5], [1], [8, 9], [16, 17], [32, 33], [64, 2, 64]])
@pytest.mark.parametrize("idx_dtype", [torch.int64, torch.int32])
def test_batch_equals_hops(cuda, fanouts, idx_dtype, monkeypatch):
    import cxgnncomp
    import cxgnncomp_backend as be
    from cxgnncomp import synthetic
    for n, und, seeds in ((4099, 30000, 130), (33, 70, 7), (70000, 400000, 1)):
        ptr, idx = synthetic.powerlaw_graph(n, und, seed=len(fanouts))
        p, i = ptr.cuda(), idx.cuda().to(idx_dtype)
        s = torch.randperm(n, generator=torch.Generator().manual_seed(n))[:seeds].cuda()
        sampler = cxgnncomp.NeighborSampler(p, i, fanouts)
        got = [sampler.sample(s, seed=k) for k in (5, 6)]
        assert bool((sampler.local_of == -1).all()) and not bool(sampler._marks.any())
        with monkeypatch.context() as m:
            m.setattr(be, "sample_batch_fits", lambda *a: False)
            want = [sampler.sample(s, seed=k) for k in (5, 6)]
        for g, w in zip(got, want):
            assert g[3] == w[3] and g[4] == w[4]
            for a, b in zip(g[:3], w[:3]):
                assert torch.equal(a, b)


@pytest.mark.parametrize("fanouts", [[15, 10], [40]])
def test_repeated_seeds(cuda, fanouts, monkeypatch):
    """Every seed keeps a row of its own: the first hop reaches more edges than a small graph has."""
    import cxgnncomp
    import cxgnncomp_backend as be
    ptr, idx = torch.tensor([0, 3, 4, 4, 6, 10]), torch.tensor([1, 2, 3, 0, 4, 4, 0, 1, 2, 3])
    sampler = cxgnncomp.NeighborSampler(ptr.cuda(), idx.cuda(), fanouts)
    seeds = torch.tensor([4, 0, 4, 2, 3] * 60)
    got = sampler.sample(seeds.cuda(), seed=1)
    assert bool((sampler.local_of == -1).all()) and not bool(sampler._marks.any())
    with monkeypatch.context() as m:
        m.setattr(be, "sample_batch_fits", lambda *a: False)
        want = sampler.sample(seeds.cuda(), seed=1)
    assert got[3] == want[3] and got[4] == want[4] and got[4][0] == 60 * (4 + 3 + 4 + 2)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    # which of a node's batch ids a neighbour gets is open
    assert torch.equal(got[0][got[2]], want[0][want[2]])


@pytest.mark.parametrize("bad", [-1, 33, 1 << 40])
@pytest.mark.parametrize("one_call", [True, False])
def test_seeds_outside_the_graph(cuda, bad, one_call, monkeypatch):
    import cxgnncomp
    import cxgnncomp_backend as be
    from cxgnncomp import synthetic
    ptr, idx = synthetic.powerlaw_graph(33, 70, seed=3)
    sampler = cxgnncomp.NeighborSampler(ptr.cuda(), idx.cuda(), [4, 3])
    seeds = torch.tensor([5, 30, 2, 9])
    if not one_call:
        monkeypatch.setattr(be, "sample_batch_fits", lambda *a: False)
    want = sampler.sample(seeds.cuda(), seed=2)
    with pytest.raises(RuntimeError, match="seeds must be node ids"):
        sampler.sample(torch.cat([seeds, torch.tensor([bad])]).cuda(), seed=2)
    assert bool((sampler.local_of == -1).all()) and not bool(sampler._marks.any())
    for a, b in zip(sampler.sample(seeds.cuda(), seed=2), want):
        assert torch.equal(a, b) if isinstance(a, torch.Tensor) else a == b
