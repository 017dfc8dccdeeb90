"""FP32 translations (sfmm_f32.cuh): every block count and remainder of the
lane layout, both group sizes, uniform and mixed orders, scaled shifts, against
the FP64 oracle on the FP32-rounded inputs.

Tolerance: 2^-24 per rounding, about 4 d roundings of the row's norm along the
transforms and the z-translation of degree d <= P, growing by 1.35 per degree
for M2M above order 16 (as in every arithmetic): the 2e-5 that the FP32 tests
of this repository ask at orders up to 24, 5e-5 above."""
import numpy as np
import pytest

from helpers import norm_weights, rel_err, run_device

pytestmark = pytest.mark.gpu

OPS = ("m2m", "m2l", "l2l")


@pytest.mark.parametrize("group", [4, 8])
@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("P", [1, 2, 3, 4, 5, 8, 9, 12, 13, 16, 17, 20, 21, 24, 25, 28])
def test_orders_and_remainders(native, oracle, op, P, group):
    from inputs import make_batch

    ctx = native.Context(P, "f32")
    ctx.set_group(native.PLAIN, group, order_bound=P)
    w = norm_weights(P, "M" if op == "m2m" else "L")
    for spec in (P, (1, P)):
        b = make_batch(np.random.default_rng(100 * P + OPS.index(op)), op, spec, spec, 37, nq=6)
        src = b["src"].astype(np.float32)
        ref = np.zeros_like(b["dst"])
        oracle.naive(op, src.astype(np.float64), b["Pin"], ref, b["Pout"], b["xyz"])
        pad = ((0, 0), (0, P * (P + 1) - src.shape[1]))
        src, ref = np.pad(src, pad), np.pad(ref, pad)
        got = run_device(ctx, op, native.PLAIN, src, np.zeros_like(src), b["Pin"], b["Pout"], b["xyz"], order_bound=P)
        assert rel_err(got, ref, w) < (2e-5 if P <= 24 else 5e-5), spec
