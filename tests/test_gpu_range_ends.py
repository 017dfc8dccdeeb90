"""Translations at the ends of the FP64 range: shifts next to the z axis and
coefficients next to the smallest doubles."""
import numpy as np
import pytest

from helpers import norm_weights, rel_err, run_device

pytestmark = pytest.mark.gpu

OPS = ("m2m", "m2l", "l2l")


@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("dtype,tol", [("f64", 1e-12), ("f32", 2e-5)])
def test_shifts_next_to_the_z_axis(native, op, dtype, tol):
    """A transverse part of t |z|, t <= 2^-64, changes the result by less than
    a rounding at most, whatever becomes of the squares of its components
    (from t = 2^-511 on they leave the FP64 range beside z^2): the results are
    those of the shift along the axis, to the tolerance that the tests against
    the oracle ask of either."""
    P, S = 10, 110
    rng = np.random.default_rng(5)
    t = np.array([2.0 ** -64, 2.0 ** -150, 1.2 * 2.0 ** -500, 2.0 ** -511, 1.37e-160, 1.2 * 2.0 ** -537, 2.0 ** -600,
                  2.0 ** -900])
    dirs = np.array([[1, 0], [0, -1], [0.6, 0.8], [-1, 2.0 ** -30]])
    xy = (t[:, None, None] * dirs).reshape(-1, 2)
    z = np.array([2.5, -0.75, 1e10])[:, None] * np.ones(len(xy))
    z[:, ::2] /= 2
    sh = np.stack([np.broadcast_to(xy[:, 0], z.shape) * abs(z), np.broadcast_to(xy[:, 1], z.shape) * abs(z), z], -1)
    sh = sh[:2].reshape(-1, 3) if dtype == "f32" else sh.reshape(-1, 3)  # 1e10^19 is no FP32 number
    n = len(sh)
    w, wo = norm_weights(P, "L" if op == "l2l" else "M"), norm_weights(P, "M" if op == "m2m" else "L")
    deg = np.array([d for d in range(P) for _ in range(2 * (d + 1))])
    length = abs(sh[:, 2:])  # expansions at the length scale of their shift
    src = rng.normal(size=(n, S)) / w * length ** (-deg - 1 if op == "l2l" else deg)
    src = src.astype(np.float64 if dtype == "f64" else np.float32)
    for d in range(P):
        src[:, (d + 1) ** 2] = 0
    p = np.full(n, P, np.uint32)
    ctx = native.Context(P, dtype)
    axis = sh * np.array([0, 0, 1])
    got, ref = (run_device(ctx, op, native.PLAIN, src, np.zeros_like(src), p, p, s).astype(np.float64) for s in (sh, axis))
    back = length ** (-deg if op == "m2m" else deg + 1)
    assert rel_err(got * back, ref * back, wo) < tol
