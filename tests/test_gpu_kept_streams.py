"""What is kept per graph (transposed graphs, combined indices, destinations) and taken by another stream than the one that built
it, by a capture, and from a capture: the builder is held up, so that whoever does not wait reads what is not there yet."""
import pytest
import torch

from helpers import random_csr, randn

pytestmark = pytest.mark.gpu

N, WIDTH = 3000, 32


def _graph(seed):
    return tuple(t.cuda() for t in random_csr(N, N, 6, seed=seed))


def _aggregation(kind, ptr, idx):
    import cxgnncomp
    import cxgnncomp_backend as be
    g = randn((N, WIDTH), 2).cuda()
    if kind == "gat":
        torch.manual_seed(1)
        conv, x = cxgnncomp.MyGATConv(WIDTH, 8, heads=4, concat=True).cuda(), randn((N, WIDTH), 1).cuda().requires_grad_(True)
        return lambda: torch.autograd.grad(conv(x, ptr, idx, N, N, idx.shape[0]), [x], g)[0]
    if kind == "relation":
        rel = torch.randint(0, 3, (idx.shape[0],), generator=torch.Generator().manual_seed(3)).int().cuda()
        x = randn((3 * N, WIDTH), 1).cuda().requires_grad_(True)
        return lambda: torch.autograd.grad(be.aggr_rel(x, ptr, idx, rel, N, 3), [x], g)[0]
    if kind == "sddmm":
        a, b = randn((N, 2, WIDTH), 1).cuda(), randn((N, WIDTH), 4).cuda()
        return lambda: be.run_sddmm_vertex_centric(ptr, idx, a, b, N)
    x, val = randn((N, WIDTH), 1).cuda().requires_grad_(True), randn((idx.shape[0],), 3).cuda()
    if kind == "value":
        return lambda: torch.autograd.grad(be.sage_sum_forward_edge_value(x, ptr, idx, val, N), [x], g)[0]
    fn = be.sage_sum_forward if kind == "sum" else be.sage_mean_forward
    return lambda: torch.autograd.grad(fn(x, ptr, idx, N), [x], g)[0]


def _same(a, b):
    # the GAT layer's gradient of the scores adds with atomics, in no fixed order: sums of at most a few dozen terms
    return torch.equal(a, b) or float((a - b).norm()) <= 1e-5 * float(b.norm())


@pytest.mark.parametrize("kind", ["sum", "mean", "value", "gat", "relation", "sddmm"])
def test_other_stream_waits_for_the_builder(cuda, kind):
    import cxgnncomp_backend as be
    run = _aggregation(kind, *_graph(1))
    want = run()
    torch.cuda.synchronize()
    be.forget_graphs()
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(first):
        torch.cuda._sleep(100_000_000)
        a = run()  # builds
    with torch.cuda.stream(second):
        b = run()  # takes
        torch.cuda._sleep(20_000_000)
        c = run()
    be.forget_graphs()  # while `second` is still to read it
    with torch.cuda.stream(first):
        waste = [torch.full((1 << 16,), -1, dtype=torch.int64, device="cuda") for _ in range(16)]
    torch.cuda.synchronize()
    assert len(waste) == 16 and _same(a, want) and _same(b, want) and _same(c, want)


@pytest.mark.parametrize("kind", ["sum", "mean", "relation"])
@pytest.mark.parametrize("kept_before", [False, True])
def test_capture(cuda, kind, kept_before):
    """A capture takes what is kept; what it builds itself is not there for others, who come before it is replayed."""
    import cxgnncomp_backend as be
    run = _aggregation(kind, *_graph(2))
    want = run()
    torch.cuda.synchronize()
    if not kept_before:
        be.forget_graphs()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = run()
    assert _same(run(), want)
    graph.replay()
    torch.cuda.synchronize()
    assert _same(got, want) and _same(run(), want)
    be.forget_graphs()


@pytest.mark.parametrize("kind", ["sum", "mean", "relation", "gat"])
def test_replay_after_others(cuda, kind):
    """What a capture has taken or used as scratch stays its own: nine other graphs, larger calls on its stream and other tensors
    come between the capture and its replay."""
    import cxgnncomp_backend as be
    be.forget_graphs()
    side = torch.cuda.Stream()
    run = _aggregation(kind, *_graph(3))
    others = [_aggregation(kind, *_graph(10 + i)) for i in range(9)]
    large = [t.cuda() for t in random_csr(40_000, 40_000, 30, seed=4)]
    with torch.cuda.stream(side):
        want = run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        got = run()
    with torch.cuda.stream(side):
        for other in others:
            other()
        be.sage_sum_forward(randn((40_000, 256), 5).cuda(), *large, 40_000)
        waste = [torch.full((1 << k,), 7, dtype=torch.int64, device="cuda") for k in range(9, 20) for _ in range(8)]
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert _same(got, want) and all(bool((w == 7).all()) for w in waste)
    del graph
    be.forget_graphs()
