"""Plain FP64 in 60-bit block fixed point (sfmm_fx.cuh): every block count and
remainder of its lane layout against the FP64 oracle, exact scaling by powers
of two, and non-finite inputs.

Tolerance: 1e-12 in the orthonormal basis, what the other tests of plain FP64
ask (the kernel is no less accurate than FP64 arithmetic, whose own error
grows to 7e-14 at order 28 for M2M)."""
import numpy as np
import pytest

from helpers import norm_weights, rel_err, run_device

pytestmark = pytest.mark.gpu

OPS = ("m2m", "m2l", "l2l")


@pytest.mark.parametrize("group", [4, 8])
@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("P", [1, 2, 3, 4, 5, 8, 9, 12, 13, 16, 17, 20, 21, 24, 25, 28, 29, 32])
def test_orders_and_remainders(native, oracle, op, P, group):
    """Uniform order P, and orders mixed up to P (source and target apart),
    37 translations (a partial tile and a partial warp)."""
    from inputs import make_batch

    ctx = native.Context(P, "f64")
    ctx.set_group(native.PLAIN, group, order_bound=P)
    w = norm_weights(P, "M" if op == "m2m" else "L")
    for spec in (P, (1, P)):
        b = make_batch(np.random.default_rng(100 * P + OPS.index(op)), op, spec, spec, 37, nq=6)
        ref = b["dst"].copy()
        oracle.naive(op, b["src"], b["Pin"], ref, b["Pout"], b["xyz"])
        pad = P * (P + 1) - b["src"].shape[1]
        src, dst = (np.pad(b[k], ((0, 0), (0, pad))) for k in ("src", "dst"))
        got = run_device(ctx, op, native.PLAIN, src, dst, b["Pin"], b["Pout"], b["xyz"], order_bound=P)
        assert rel_err(got - dst, np.pad(ref - b["dst"], ((0, 0), (0, pad))), w) < 1e-12, spec


@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("P", [7, 18])
def test_powers_of_two_are_exact(native, op, P):
    """Sources times 2^k give results times 2^k, bit for bit."""
    rng = np.random.default_rng(P)
    n, S = 33, P * (P + 1)
    src = rng.normal(size=(n, S))
    sh = rng.normal(size=(n, 3))
    p = np.full(n, P, np.uint32)
    ctx = native.Context(P, "f64")
    base = run_device(ctx, op, native.PLAIN, src, np.zeros((n, S)), p, p, sh)
    for k in (-500, 300):
        got = run_device(ctx, op, native.PLAIN, np.ldexp(src, k), np.zeros((n, S)), p, p, sh)
        assert np.array_equal(got, np.ldexp(base, k)), k


@pytest.mark.parametrize("op", OPS)
def test_non_finite_inputs_stay_in_their_translation(native, op):
    """A NaN, an infinity, a non-finite shift and (M2L) a zero shift make the
    degrees of their own target non-finite that depend on them, and leave
    every other target as it is; the imaginary part at m = 0, which is zero in
    every expansion, is not read as a number."""
    P, n = 9, 40
    S = P * (P + 1)
    rng = np.random.default_rng(3)
    src = rng.normal(size=(n, S))
    sh = rng.normal(size=(n, 3))
    for d in range(P):
        src[:, (d + 1) ** 2] = 0.0
    p = np.full(n, P, np.uint32)
    ctx = native.Context(P, "f64")
    clean = run_device(ctx, op, native.PLAIN, src, np.zeros((n, S)), p, p, sh)
    bad = [5, 6, 7, 20] + ([21] if op == "m2l" else [])
    s2, h2 = src.copy(), sh.copy()
    s2[5, 20] = np.nan  # degree 4
    s2[6, 21] = np.inf
    h2[7, 1] = np.nan
    h2[20, 0] = np.inf
    if op == "m2l":
        h2[21] = 0.0
    for d in range(P):
        s2[30, (d + 1) ** 2] = np.nan
    got = run_device(ctx, op, native.PLAIN, s2, np.zeros((n, S)), p, p, h2)
    keep = [i for i in range(n) if i not in bad]
    assert np.array_equal(got[keep], clean[keep])
    # degrees that a source's degree 4 reaches: >= 4 (M2M), all (M2L), <= 4 (L2L)
    lo, hi = {"m2m": (4, P), "m2l": (0, P), "l2l": (0, 5)}[op]
    for i in (5, 6):
        assert not np.isfinite(got[i, lo * (lo + 1):hi * (hi + 1)]).any()
        assert np.array_equal(got[i, : lo * (lo + 1)], clean[i, : lo * (lo + 1)])
        assert np.array_equal(got[i, hi * (hi + 1):], clean[i, hi * (hi + 1):])
    for i in bad[2:]:
        assert not np.isfinite(got[i]).any()
