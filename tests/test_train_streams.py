"""red_mlp_grad on several streams and threads at once, and captured in graphs: each
call's gradient and loss are the bits of the call alone (the per-CTA partial gradients
of one call are not another's)."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


class Job:
    """A network, a batch and the result of the call alone."""

    def __init__(self, rg, rows, seed):
        g = torch.Generator().manual_seed(seed)
        n = rg.lib.load().red_mlp_param_count()
        self.rg, self.rows, self.n = rg, rows, n
        self.w = (0.2 * torch.randn(n, generator=g)).bfloat16().cuda()
        self.x = torch.randn(rows, 12, generator=g).cuda()
        self.t = torch.randn(rows, generator=g).cuda()
        self.grad, self.loss = self.out()
        self.call(self.grad, self.loss, torch.cuda.current_stream())
        torch.cuda.synchronize()

    def out(self):
        return torch.zeros(self.n, device="cuda"), torch.zeros(1, device="cuda")

    def call(self, grad, loss, stream):
        self.rg.lib.mlp_grad(self.w.data_ptr(), self.x.data_ptr(), self.t.data_ptr(), self.rows, grad.data_ptr(),
                             loss.data_ptr(), stream.cuda_stream)

    def same(self, grad, loss):
        return torch.equal(grad, self.grad) and torch.equal(loss, self.loss)


def jobs(rg):
    return [Job(rg, rows, k) for k, rows in enumerate((2048, 30000, 100, 9000))]


def test_streams(rg):
    js = jobs(rg)
    streams = [torch.cuda.Stream() for _ in js]
    outs = [[j.out() for _ in range(100)] for j in js]
    torch.cuda.synchronize()
    for k in range(100):
        for j, s, o in zip(js, streams, outs):
            j.call(*o[k], s)
    torch.cuda.synchronize()
    assert all(j.same(*x) for j, o in zip(js, outs) for x in o)


def test_threads(rg):
    js = jobs(rg)
    outs = [[j.out() for _ in range(100)] for j in js]
    torch.cuda.synchronize()
    failed = []

    def work(j, o):
        try:
            s = torch.cuda.Stream()
            for x in o:
                j.call(*x, s)
            s.synchronize()
        except Exception as e:   # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=work, args=a) for a in zip(js, outs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed and all(j.same(*x) for j, o in zip(js, outs) for x in o)


def test_captured(rg):
    """Replays beside calls on another stream."""
    a, b = Job(rg, 20000, 1), Job(rg, 25000, 2)
    ga, la = a.out()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        a.call(ga, la, torch.cuda.current_stream())
    outs = [b.out() for _ in range(60)]
    s, r = torch.cuda.Stream(), torch.cuda.Stream()
    ok = torch.zeros(1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    for o in outs:
        with torch.cuda.stream(r):
            graph.replay()
            ok += ((ga == a.grad).all() & (la == a.loss).all()).long()
        b.call(*o, s)
    torch.cuda.synchronize()
    assert int(ok) == len(outs) and all(b.same(*o) for o in outs)
