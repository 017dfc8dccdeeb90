"""Evaluation on both sides of the lines between its forms (one or four lanes
per point, gradients from pairings or per point), against the FP64 kernel.

Tolerance: 1e-12 of the largest value, what tests/test_gpu_leaf_routes.py asks
of the same forms."""
import pytest

from helpers import S_of

pytestmark = pytest.mark.gpu

# (points, expansions): four lanes with and without pairings, one lane with and
# without (45 000 is beyond both lines on 152 SMs), an odd count of each
CALLS = [(513, 64), (511, 64), (301, 300), (19_400, 1000), (19_600, 1000), (38_800, 1000), (45_001, 5000), (45_000, 45_000)]


@pytest.mark.parametrize("P", [2, 3, 4, 11, 12, 15, 16, 24])
def test_both_sides_of_the_lines(native, P):
    import torch

    opt = dict(dtype=torch.float64, device="cuda:0")
    g = torch.Generator(device="cuda:0")
    g.manual_seed(P)
    S, most = S_of(P), 45_001
    cen = torch.rand(most, 3, generator=g, **opt)
    src = torch.randn(most, 3, 3, generator=g, **opt)
    src = src / src.norm(dim=2, keepdim=True) * (1 + torch.rand(most, 3, 1, generator=g, **opt))
    ctx = native.Context(P, "f64")
    E = torch.zeros(most, S, **opt)
    ctx.p2x(1, most, 3, torch.rand(most, 3, generator=g, **opt) - 0.5, (cen[:, None] + src).contiguous(), cen, E, S)
    few = 200  # compared with the FP64 kernel: fewer than one point per four expansions
    for npts, nexp in CALLS:
        box = torch.randint(0, nexp, (npts,), device="cuda:0", generator=g).to(torch.int32)
        u = torch.randn(npts, 3, generator=g, **opt)
        pos = (cen[box.long()] + 0.4 * u / u.norm(dim=1, keepdim=True)).contiguous()
        out = []
        for n, k in ((npts, nexp), (few, most)):
            for gradient in (True, False):
                pot = torch.zeros(n, **opt)
                grad = torch.zeros(n, 3, **opt) if gradient else None
                ctx.evaluate(0, n, pos[:n].contiguous(), E, S, k, cen, pot, gradient=grad, box=box[:n].contiguous())
                out.append((pot, grad))
        torch.cuda.synchronize()
        (p1, g1), (p2, _), (p0, g0), _ = out
        for a, b in ((p1, p0), (p2, p0), (g1, g0)):
            assert float((a[:few] - b).abs().max()) <= 1e-12 * float(b.abs().max()), (npts, nexp)
