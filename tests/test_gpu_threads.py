"""Several threads on one stream: the launches of a call hand its stream's scratch buffer on to each other, so no launch of
another thread's call may come between them, whether that one holds the interpreter's lock or is a backward of autograd."""
import threading
import time

import pytest
import torch

from helpers import random_csr, randn

pytestmark = pytest.mark.gpu


def test_calls_wait_for_the_buffer(cuda):
    import cxgnncomp_backend as be
    ptr, idx = random_csr(300, 300, 8, seed=1, hub=500)
    x = randn((300, 64), 2).cuda().requires_grad_()
    p, i = ptr.cuda(), idx.cuda()
    want = be.sage_sum_forward(x, p, i, 300)
    (gx,) = torch.autograd.grad(want, x, want.detach())
    loss = be.sage_sum_forward(x, p, i, 300)
    done = []
    calls = [lambda: done.append(be.sage_sum_forward(x, p, i, 300)),
             lambda: done.append(be.column_sum(want.detach())),
             lambda: done.append(torch.autograd.grad(loss, x, want.detach())[0])]
    threads = [threading.Thread(target=c) for c in calls]
    with be._workspace(x.device, 1024) as ws:
        assert ws.numel() >= 1024
        for t in threads:
            t.start()
        time.sleep(0.3)
        assert not done
    for t in threads:
        t.join(60)
        assert not t.is_alive()
    assert len(done) == 3
    assert any(t.shape == want.shape and torch.equal(t, want) for t in done) and any(torch.equal(t, gx) for t in done)


def test_threads_on_one_stream(cuda):
    import cxgnncomp_backend as be
    jobs = []
    for k, (n, f) in enumerate([(4000, 64), (900, 100), (2500, 47)]):
        ptr, idx = random_csr(n, n, 12, seed=k, hub=30000)
        x = randn((n, f), k + 10).cuda().requires_grad_()
        jobs.append((x, ptr.cuda(), idx.cuda(), n))

    def step(job):
        x, p, i, n = job
        y = be.sage_mean_forward(x, p, i, n)
        return y.detach(), torch.autograd.grad(y, x, y.detach())[0], be.column_sum(y.detach())

    want = [step(j) for j in jobs]
    wrong = []

    def work(k):
        for _ in range(40):
            if not all(torch.equal(a, b) for a, b in zip(step(jobs[k]), want[k])):
                wrong.append(k)

    threads = [threading.Thread(target=work, args=(k % 3,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
        assert not t.is_alive()
    assert not wrong
