"""Launch shapes pinned or tuned for one precision mode leave the others alone."""
import numpy as np
import pytest

from helpers import run_device

pytestmark = pytest.mark.gpu


def test_pins_belong_to_their_mode(native):
    """split_ff runs plain FP64's kernel, but a group size pinned for it is not
    plain's (nor the other way round).  Powers of e^{i alpha} are formed in
    steps of the group's rows, so the last bits tell the group size."""
    P, n = 10, 60
    S = P * (P + 1)
    rng = np.random.default_rng(2)
    src, sh, p = rng.normal(size=(n, S)), rng.normal(size=(n, 3)) + 2, np.full(n, P, np.uint32)

    def bits(ctx, mode):
        return run_device(ctx, "m2l", mode, src, np.zeros((n, S)), p, p, sh)

    four, eight = (native.Context(P, "f64") for _ in range(2))
    for ctx, g in ((four, 4), (eight, 8)):
        for mode in (native.PLAIN, native.SPLIT_FF):
            ctx.set_group(mode, g, order_bound=P)
    want = {4: bits(four, native.PLAIN), 8: bits(eight, native.PLAIN)}
    assert not np.array_equal(want[4], want[8])
    for mode, other in ((native.PLAIN, native.SPLIT_FF), (native.SPLIT_FF, native.PLAIN)):
        ctx = native.Context(P, "f64")
        ctx.set_group(mode, 4, order_bound=P)
        ctx.set_group(other, 8, order_bound=P)
        assert np.array_equal(bits(ctx, mode), want[4])
        assert np.array_equal(bits(ctx, other), want[8])
        ctx.set_group(mode, 4, order_bound=P)
        ctx.tune("m2l", other, n=4096, order_bound=P)
        assert np.array_equal(bits(ctx, mode), want[4])
