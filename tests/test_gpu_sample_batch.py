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
