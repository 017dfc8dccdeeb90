"""The forms of P2M/P2L and of L2P/M2P that a call's size chooses between give
the same sums: lanes shared per expansion or per point, equal or ragged
charge counts, gradients from prepared pairings or formed per point.

Tolerances: each P2M form is within 6.0e-14 of the sum of its terms' absolute
bounds (what tests/test_gpu_p2x.py measures), so two differ by 1.2e-13 at most;
evaluation is compared with the FP64 kernel, 1e-12 of the largest value."""
import numpy as np
import pytest

from helpers import S_of, p2x_abs_scale

pytestmark = pytest.mark.gpu

ORDERS = [1, 2, 3, 4, 5, 8, 9, 13, 16, 17, 24, 25, 32]


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("P", ORDERS)
def test_p2x_forms(native, P, kind):
    import torch

    dev = "cuda:0"
    g = torch.Generator(device=dev)
    g.manual_seed(P)
    S, many, nq = S_of(P), 12_000, 5
    d = torch.randn(many, nq, 3, dtype=torch.float64, device=dev, generator=g)
    pos = d / d.norm(dim=2, keepdim=True) * (0.2 + 0.3 * torch.rand(many, nq, 1, dtype=torch.float64, device=dev, generator=g))
    q = torch.rand(many, nq, dtype=torch.float64, device=dev, generator=g) - 0.5
    cen = 0.01 * torch.rand(many, 3, dtype=torch.float64, device=dev, generator=g)
    off = (torch.arange(many + 1, device=dev) * nq).to(torch.int32)
    ctx = native.Context(P, "f64")
    out = [torch.zeros(many, S, dtype=torch.float64, device=dev) for _ in range(3)]
    ctx.p2x(kind, many, nq, q, pos, cen, out[0], S)            # one group per expansion
    ctx.p2x_ragged(kind, many, off, q, pos, cen, out[1], S)    # ragged counts
    few = 37
    ctx.p2x_ragged(kind, few, off, q, pos, cen, out[2], S)     # few expansions
    torch.cuda.synchronize()
    scale = torch.as_tensor(p2x_abs_scale(P, kind, q[:400].cpu().numpy(), pos[:400].cpu().numpy(), cen[:400].cpu().numpy()),
                            device=dev)
    scale = torch.where(scale > 0, scale, torch.ones_like(scale))
    assert float(((out[1][:400] - out[0][:400]).abs() / scale).max()) < 1.2e-13
    assert float(((out[2][:few] - out[0][:few]).abs() / scale[:few]).max()) < 1.2e-13
    assert not out[2][few:].any()
    # counts of 0 .. 2 nq, the same charges for the expansions that keep theirs
    cnt = torch.randint(0, 2 * nq + 1, (many,), device=dev, generator=g)
    cnt[:3] = torch.tensor([0, 1, 2 * nq], device=dev)
    roff = torch.zeros(many + 1, dtype=torch.int64, device=dev)
    roff[1:] = torch.cumsum(cnt, 0)
    k = int(roff[-1])
    rep = torch.repeat_interleave(torch.arange(many, device=dev), cnt)
    rq = torch.rand(k, dtype=torch.float64, device=dev, generator=g) - 0.5
    rp = pos.reshape(-1, 3)[torch.arange(k, device=dev) % (many * nq)].contiguous()
    a, b = torch.zeros_like(out[0]), torch.zeros_like(out[0])
    ctx.p2x_ragged(kind, many, roff.to(torch.int32), rq, rp, cen, a, S)
    for i in range(3):  # one expansion at a time: the few-expansions form
        s = slice(int(roff[i]), int(roff[i + 1]))
        if s.stop > s.start:
            one = torch.tensor([0, s.stop - s.start], dtype=torch.int32, device=dev)
            ctx.p2x_ragged(kind, 1, one, rq[s].contiguous(), rp[s].contiguous(), cen[i:i + 1].contiguous(), b[i:i + 1], S)
            sc = torch.as_tensor(p2x_abs_scale(P, kind, rq[s].cpu().numpy()[None], rp[s].cpu().numpy()[None],
                                               cen[i:i + 1].cpu().numpy()), device=dev)
            sc = torch.where(sc > 0, sc, torch.ones_like(sc))
            assert float(((a[i] - b[i]).abs() / sc[0]).max()) < 1.2e-13
    assert not a[0].any()


@pytest.mark.parametrize("P", ORDERS)
def test_evaluation_forms(native, P):
    import torch

    dev = "cuda:0"
    g = torch.Generator(device=dev)
    g.manual_seed(100 + P)
    S = S_of(P)
    ctx = native.Context(P, "f64")

    def rand(*s):
        return torch.rand(*s, dtype=torch.float64, device=dev, generator=g)

    nbox = 64
    cen = rand(nbox, 3)
    # locals of charges one to two units away, multipoles of charges inside
    src = torch.randn(nbox, 8, 3, dtype=torch.float64, device=dev, generator=g)
    src = src / src.norm(dim=2, keepdim=True)
    loc, mul = (torch.zeros(nbox, S, dtype=torch.float64, device=dev) for _ in range(2))
    ctx.p2x(1, nbox, 8, rand(nbox, 8) - 0.5, (cen[:, None] + src * (1 + rand(nbox, 8, 1))).contiguous(), cen, loc, S)
    ctx.p2x(0, nbox, 8, rand(nbox, 8) - 0.5, (cen[:, None] + 0.3 * src).contiguous(), cen, mul, S)
    n = 45_000  # one lane per point; the first 200 alone take several
    box = torch.randint(0, nbox, (n,), device=dev, generator=g).to(torch.int32)
    u = torch.randn(n, 3, dtype=torch.float64, device=dev, generator=g)
    u = u / u.norm(dim=1, keepdim=True)
    near = (cen[box.long()] + 0.3 * rand(n, 1) * u).contiguous()
    far = (cen[box.long()] + (1 + rand(n, 1)) * u).contiguous()

    def run(kind, k, expansions, grad):
        pot = torch.zeros(k, dtype=torch.float64, device=dev)
        gr = torch.zeros(k, 3, dtype=torch.float64, device=dev) if grad else None
        E = loc if kind == 0 else mul
        E = torch.cat([E, torch.zeros(expansions - nbox, S, dtype=torch.float64, device=dev)]) if expansions > nbox else E
        c = torch.cat([cen, torch.zeros(expansions - nbox, 3, dtype=torch.float64, device=dev)]) if expansions > nbox else cen
        ctx.evaluate(kind, k, (near if kind == 0 else far)[:k].contiguous(), E, S, expansions, c, pot, gradient=gr,
                     box=box[:k].contiguous())
        torch.cuda.synchronize()
        return pot, gr

    m = 200
    for kind in (0, 1):
        grad = kind == 0
        ref = run(kind, m, 4 * m + 1, grad)  # fewer than one point per four expansions: FP64
        # pairings prepared (one lane, four lanes), formed per point (four points per expansion not reached)
        for got in (run(kind, n, nbox, grad), run(kind, 4 * nbox, nbox, grad), run(kind, m, m, grad), run(kind, m, nbox, False)):
            for a, b in zip(got, ref):
                if a is not None and b is not None:
                    assert float((a[:m] - b).abs().max()) <= 1e-12 * float(b.abs().max()), kind
