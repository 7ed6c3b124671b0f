"""Infinities, NaN and values above bf16's range (3.39e38) through the layers' linear transform and its gradients: what an fp32
chain gives, element for element, and nothing else touched."""
import pytest
import torch

from helpers import randn

pytestmark = pytest.mark.gpu
INF, NAN, BIG = float("inf"), float("nan"), 3.4e38


def same(got, want, tol):
    """Infinities and NaN in the same places; elsewhere within tol of the largest value of the row's scale."""
    got, want = got.cpu().double(), want.float().double()  # float(): what does not fit fp32 is an infinity
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.isinf(), want.isinf()) and torch.equal(got[got.isinf()], want[want.isinf()])
    ok = want.isfinite()
    scale = torch.where(ok, want.abs(), 0).amax(1, keepdim=True).clamp(min=1e-30)
    assert float(((got - want).abs() / scale)[ok].max()) < tol


def planted(t, seed, kinds=(INF, -INF, NAN, BIG, -BIG)):
    """Some values of every kind, each in a row and a column of its own: with two values at the end of the range in one sum
    an fp32 result depends on the order of the additions (an infinity on the way or not), and the float64 one says nothing."""
    rows = torch.randperm(t.shape[0], generator=torch.Generator().manual_seed(seed))[:5].tolist()
    for j, (r, v) in enumerate(zip(rows, kinds)):
        t[r, j % t.shape[1]] = v
    return t


@pytest.mark.parametrize("m,k,n", [(5, 4, 3), (128, 32, 16), (300, 36, 47), (1000, 128, 128), (9, 64, 256)])
@pytest.mark.parametrize("where", ["x", "w", "both"])
def test_product(cuda, m, k, n, where):
    import cxgnncomp_backend as be
    x, w = randn((m, k), 1), randn((max(n, 5), k), 2)[:n] * 0.25
    w[:, ::3] = (w[:, ::3] * 4).round() / 4  # exact in bf16, zeros among them: lower terms that are zero
    kinds = (INF, -INF, NAN) if where == "both" else (INF, -INF, NAN, BIG, -BIG)
    if where != "w":
        planted(x, 3, kinds)
    if where != "x" and n >= 5:
        planted(w, 4, kinds)
    b, add = randn((n,), 5), randn((m, n), 6)
    want = x.double() @ w.double().t() + b.double()
    with torch.no_grad():
        same(be.linear(x.cuda(), w.cuda(), b.cuda()), want, 4e-6)
        same(be.linear(x.cuda(), w.cuda(), b.cuda(), add.cuda()), want + add.double(), 4e-6)


@pytest.mark.parametrize("m,k,n", [(40, 16, 8), (700, 36, 64), (3000, 200, 132)])
@pytest.mark.parametrize("where", ["x", "g"])
def test_gradients(cuda, m, k, n, where):
    import cxgnncomp_backend as be
    x, w, g = randn((m, k), 1), randn((n, k), 2), randn((m, n), 3)
    planted(x if where == "x" else g, 7)
    xd, wd = x.cuda().requires_grad_(), w.cuda().requires_grad_()
    gx, gw = torch.autograd.grad(be.linear(xd, wd, same_bits=True), [xd, wd], g.cuda())
    same(gx, g.double() @ w.double(), 4e-6)
    same(gw, g.double().t() @ x.double(), 4e-6)
