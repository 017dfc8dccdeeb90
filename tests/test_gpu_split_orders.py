"""Split precision (sfmm_split.cuh): every block count and remainder of both
group sizes, uniform and mixed orders, against the FP64 oracle, at the mode's
1e-7 contract in the orthonormal basis."""
import numpy as np
import pytest

from helpers import norm_weights, rel_err, run_device

pytestmark = pytest.mark.gpu

OPS = ("m2m", "m2l", "l2l")


@pytest.mark.parametrize("group", [4, 8])
@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("P", [1, 2, 4, 5, 8, 9, 12, 13, 16, 17, 18, 20, 21, 24, 25, 28])
def test_orders_and_remainders(native, oracle, op, P, group):
    from inputs import make_batch

    ctx = native.Context(P, "f64")
    ctx.set_group(native.SPLIT, group, order_bound=P)
    w = norm_weights(P, "M" if op == "m2m" else "L")
    for spec in (P, (1, P)):
        b = make_batch(np.random.default_rng(100 * P + OPS.index(op)), op, spec, spec, 37, nq=6)
        ref = np.zeros_like(b["dst"])
        oracle.naive(op, b["src"], b["Pin"], ref, b["Pout"], b["xyz"])
        pad = ((0, 0), (0, P * (P + 1) - ref.shape[1]))
        src, ref = np.pad(b["src"], pad), np.pad(ref, pad)
        got = run_device(ctx, op, native.SPLIT, src, np.zeros_like(src), b["Pin"], b["Pout"], b["xyz"], order_bound=P)
        assert rel_err(got, ref, w) < 1e-7, spec
