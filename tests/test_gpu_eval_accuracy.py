"""Rounding error of the float-float evaluation over many points, against the
FP64 kernel on the same expansions.

The bounds are 3% above the figures of the form that multiplies each
coefficient out at every point (norm of the error by the norm of the values,
300 000 points: M2P 7.36e-15 at order 12 and 9.18e-15 at 20, L2P gradients
7.00e-15 and 9.36e-15): preparing the expansions must not cost accuracy."""
import pytest

from helpers import S_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,P,bound", [(1, 12, 7.58e-15), (1, 20, 9.45e-15), (0, 12, 7.21e-15), (0, 20, 9.65e-15)])
def test_error_over_many_points(native, kind, P, bound):
    import torch

    dev = "cuda:0"
    g = torch.Generator(device=dev)
    g.manual_seed(17)
    opt = dict(dtype=torch.float64, device=dev)
    S, nbox, per = S_of(P), 1250, 32
    n = nbox * per

    def away(*shape):  # at a distance of 2 to 4 box sides
        d = torch.randn(*shape, 3, generator=g, **opt)
        return d / d.norm(dim=-1, keepdim=True) * (2 + 2 * torch.rand(*shape, 1, generator=g, **opt))

    def inside(*shape):
        return torch.rand(*shape, 3, generator=g, **opt) - 0.5

    far, near = (inside, away) if kind else (away, inside)
    cen = torch.rand(nbox, 3, generator=g, **opt)
    box = torch.arange(nbox, device=dev).repeat_interleave(per).to(torch.int32)
    ctx = native.Context(P, "f64")
    many = 4 * n + 1  # fewer than one point per four expansions: the FP64 kernel
    E = torch.zeros(many, S, **opt)
    cens = torch.zeros(many, 3, **opt)
    cens[:nbox] = cen
    ctx.p2x(1 - kind, nbox, 4, torch.rand(nbox, 4, generator=g, **opt) * 2 - 1,
            (cen[:, None] + far(nbox, 4)).contiguous(), cen, E, S)
    pos = (cen.repeat_interleave(per, 0) + near(n)).contiguous()
    out = []
    for nexp in (nbox, many):
        pot = torch.zeros(n, **opt)
        grad = None if kind else torch.zeros(n, 3, **opt)
        ctx.evaluate(kind, n, pos, E, S, nexp, cens, pot, gradient=grad, box=box)
        out.append(pot if kind else grad)
    torch.cuda.synchronize()
    assert float((out[0] - out[1]).norm() / out[1].norm()) < bound
