"""Translations at order bounds below their context's order (tables of another
order's strides, contexts above order 32 among them), with targets that repeat
(atomic additions), in every block count of both group sizes, against the FP64
oracle.

Tolerances in the orthonormal basis: those of the tests at equal orders, 1e-12
(plain FP64), 1e-7 (split) and 2e-5 (FP32, orders up to 24)."""
import numpy as np
import pytest

from helpers import S_of, norm_weights, rel_err, run_device

pytestmark = pytest.mark.gpu

OPS = ("m2m", "m2l", "l2l")
TOL = {("f64", "PLAIN"): 1e-12, ("f64", "SPLIT"): 1e-7, ("f32", "PLAIN"): 2e-5}


@pytest.mark.parametrize("group", [4, 8])
@pytest.mark.parametrize("dtype,mode,P", [("f64", "PLAIN", 32), ("f64", "PLAIN", 40), ("f64", "SPLIT", 28), ("f32", "PLAIN", 28)])
def test_bounds_below_the_context(native, oracle, dtype, mode, P, group):
    from inputs import make_batch

    ctx = native.Context(P, dtype)
    np_type = np.float64 if dtype == "f64" else np.float32
    for bound in (1, 3, 4, 5, 8, 9, 12, 13, 16, 17, 20, 21, 24):
        ctx.set_group(getattr(native, mode), group, order_bound=bound)
        for op in OPS:
            b = make_batch(np.random.default_rng(bound), op, (1, bound), (1, bound), 41, nq=6)
            pad = ((0, 0), (0, S_of(P) - b["src"].shape[1]))
            src = np.pad(b["src"].astype(np_type), pad)
            each = np.zeros_like(b["dst"])
            oracle.naive(op, src[:, : each.shape[1]].astype(np.float64), b["Pin"], each, b["Pout"], b["xyz"])
            tidx = np.arange(41) % 7
            ref = np.zeros((7, S_of(P)))
            np.add.at(ref, tidx, np.pad(each, pad))
            got = run_device(ctx, op, getattr(native, mode), src, np.zeros((7, S_of(P)), np_type), b["Pin"], b["Pout"],
                             b["xyz"], tidx=tidx, repeat=True, order_bound=bound)
            w = norm_weights(P, "M" if op == "m2m" else "L")
            assert rel_err(got, ref, w) < TOL[dtype, mode], (bound, op)
