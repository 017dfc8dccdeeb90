"""Evaluations recorded in a stream capture, and the scratch that they point to."""
import pytest

from helpers import S_of

pytestmark = pytest.mark.gpu

P = 12


class Batch:
    def __init__(self, npts, nexp, seed, gradient):
        import torch

        g = torch.Generator(device="cuda:0")
        g.manual_seed(seed)
        opt = dict(dtype=torch.float64, device="cuda:0")
        self.npts, self.nexp = npts, nexp
        self.cen = torch.rand(nexp, 3, generator=g, **opt)
        self.E = torch.randn(nexp, S_of(P), generator=g, **opt)
        self.box = torch.randint(0, nexp, (npts,), device="cuda:0", generator=g).to(torch.int32)
        self.pos = (self.cen[self.box.long()] + 0.1 * torch.randn(npts, 3, generator=g, **opt)).contiguous()
        self.pot = torch.zeros(npts, **opt)
        self.grad = torch.zeros(npts, 3, **opt) if gradient else None

    def evaluate(self, ctx):
        ctx.evaluate(0, self.npts, self.pos, self.E, S_of(P), self.nexp, self.cen, self.pot, gradient=self.grad, box=self.box)

    def results(self):
        import torch

        torch.cuda.synchronize()
        out = [t.clone() for t in (self.pot, self.grad) if t is not None]
        for t in (self.pot, self.grad):
            if t is not None:
                t.zero_()
        torch.cuda.synchronize()
        return out


def record(ctx, batch):
    import torch

    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        ctx.set_stream(stream.cuda_stream)
        batch.evaluate(ctx)
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    return graph


@pytest.mark.parametrize("gradient", [False, True])
def test_recorded_graph_outlives_growing_scratch(native, gradient):
    """A graph keeps the scratch it was recorded with when later calls need
    more, with or without gradients."""
    import torch

    ctx = native.Context(P, "f64")
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    small = Batch(1000, 50, 1, gradient)
    small.evaluate(ctx)
    want = small.results()
    graph = record(ctx, small)
    for nexp in (500, 5000):
        for later in (Batch(16 * nexp, nexp, nexp, True), Batch(nexp, nexp, nexp + 1, False)):
            later.evaluate(ctx)
            later.results()
        fill = torch.full((1 << 20,), float("nan"), device="cuda:0")  # what memory given back may come to hold
        graph.replay()
        got = small.results()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
        del fill


@pytest.mark.parametrize("points", [2000, 120])
def test_gradient_call_sizes_the_scratch_of_recorded_calls(native, points):
    """After one gradient call with its pairings (20 points per expansion),
    recorded calls without a gradient, and with fewer points, run the same
    kernels as calls outside a capture: the same bits, not the FP64 kernel's."""
    import torch

    warm = Batch(2000, 100, 1, True)
    later = Batch(points, 100, 2, points < 400)
    outside = native.Context(P, "f64")
    outside.set_stream(torch.cuda.current_stream().cuda_stream)
    later.evaluate(outside)
    want = later.results()
    ctx = native.Context(P, "f64")
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    warm.evaluate(ctx)
    warm.results()
    graph = record(ctx, later)
    graph.replay()
    got = later.results()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
