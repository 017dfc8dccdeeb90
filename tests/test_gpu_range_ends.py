"""Translations at the ends of the FP64 range: shifts next to the z axis and
coefficients next to the smallest doubles."""
import numpy as np
import pytest

from helpers import norm_weights, rel_err, run_device

pytestmark = pytest.mark.gpu

OPS = ("m2m", "m2l", "l2l")


def axis_error(native, op, dtype, mode, t, lengths):
    """Relative error of translations by (t |z| (u, v), z) against those by
    (0, 0, z), expansions at the length scale of their shift."""
    P, S = 10, 110
    rng = np.random.default_rng(5)
    dirs = np.array([[1, 0], [0, -1], [0.6, 0.8], [-1, 2.0 ** -30]])
    xy = (np.asarray(t)[:, None, None] * dirs).reshape(-1, 2)
    z = np.array(lengths)[:, None] * np.ones(len(xy))
    z[:, ::2] /= 2
    sh = np.stack([np.broadcast_to(xy[:, 0], z.shape) * abs(z), np.broadcast_to(xy[:, 1], z.shape) * abs(z), z], -1)
    sh = sh.reshape(-1, 3)
    n = len(sh)
    w, wo = norm_weights(P, "L" if op == "l2l" else "M"), norm_weights(P, "M" if op == "m2m" else "L")
    deg = np.array([d for d in range(P) for _ in range(2 * (d + 1))])
    length = abs(sh[:, 2:])
    src = rng.normal(size=(n, S)) / w * length ** (-deg - 1 if op == "l2l" else deg)
    src = src.astype(np.float64 if dtype == "f64" else np.float32)
    for d in range(P):
        src[:, (d + 1) ** 2] = 0
    p = np.full(n, P, np.uint32)
    ctx = native.Context(P, dtype)
    axis = sh * np.array([0, 0, 1])
    got, ref = (run_device(ctx, op, mode, src, np.zeros_like(src), p, p, s).astype(np.float64) for s in (sh, axis))
    back = length ** (-deg if op == "m2m" else deg + 1)
    return rel_err(got * back, ref * back, wo)


@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("dtype,tol", [("f64", 1e-12), ("f32", 2e-5)])
def test_shifts_next_to_the_z_axis(native, op, dtype, tol):
    """A transverse part of t |z|, t <= 2^-64, changes the result by less than
    a rounding at most, whatever becomes of the squares of its components
    (from t = 2^-511 on they leave the FP64 range beside z^2): the results are
    those of the shift along the axis, to the tolerance that the tests against
    the oracle ask of either."""
    t = [2.0 ** -64, 2.0 ** -150, 1.2 * 2.0 ** -500, 2.0 ** -511, 1.37e-160, 1.2 * 2.0 ** -537, 2.0 ** -600, 2.0 ** -900]
    lengths = [2.5, -0.75] + ([1e10] if dtype == "f64" else [])  # 1e10^19 is no FP32 number
    assert axis_error(native, op, dtype, native.PLAIN, t, lengths) < tol


@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("mode,tol", [("SPLIT", 1e-7), ("TC_TF32", 2e-5), ("TC_BF16X6", 2e-5)])
def test_shifts_next_to_the_z_axis_in_fp32_range(native, op, mode, tol):
    """The same for the modes whose geometry runs in float-float: squares lose
    their low words from t = 2^-51 on and leave the FP32 range at 2^-75."""
    t = [2.0 ** -e for e in (40, 45, 51, 56, 60, 63, 66, 69, 72, 74, 75, 76, 80, 130, 300, 900)] + [1.3e-21, 3e-22, 7e-23]
    assert axis_error(native, op, "f64", getattr(native, mode), t, [2.5, -0.75, 1e10]) < tol


@pytest.mark.parametrize("op", ("m2l", "l2l"))
def test_subnormal_sources_keep_their_digits(native, op):
    """Sources next to the smallest double, raised to normal numbers by the
    powers of a short (M2L) or long (L2L) shift, give what the same sources
    2^500 times as large give, bit for bit: only exponents differ.  Elements
    that are zero have no exponent, so one nonzero element per degree is
    enough, each in turn."""
    P, S = 4, 20
    rng = np.random.default_rng(11)
    n = 64
    src = np.zeros((n, S))
    for i in range(n):
        # L2L results take the power r^(k - n'): degrees 1 to 3 into normal results of degrees 0 to 2
        for d in range(1 if op == "l2l" else 0, P):
            m = rng.integers(0, d + 1)
            at = [d * (d + 1) + m, (d + 1) ** 2 + m][rng.integers(0, 2 if m else 1)]
            src[i, at] = np.ldexp(float(rng.integers(1, 64) * 2 + 1), int(rng.integers(-1074, -1060)))
    u = rng.normal(size=(n, 3))
    sh = np.ldexp(u / np.linalg.norm(u, axis=1, keepdims=True), -200 if op == "m2l" else 200)
    p = np.full(n, P, np.uint32)
    ctx = native.Context(P, "f64")
    zero = np.zeros((n, S))
    up = run_device(ctx, op, native.PLAIN, np.ldexp(src, 500), zero, p, p, sh)
    got = run_device(ctx, op, native.PLAIN, src, zero, p, p, sh)
    k = slice(0, S if op == "m2l" else 12)
    assert (np.abs(got[:, k]).max(1) > 0).all()
    assert np.array_equal(got[:, k], np.ldexp(up, -500)[:, k])
