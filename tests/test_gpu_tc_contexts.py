"""Tensor-core contexts of different orders side by side."""
import numpy as np
import pytest

from helpers import run_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["TC_TF32", "TC_BF16", "TC_BF16X6"])
def test_lower_order_context_leaves_the_others_working(native, mode):
    """A second context of a low order, used in between, does not shrink the
    shared memory that the first one's kernel may take."""
    prec = getattr(native, mode)
    rng = np.random.default_rng(1)

    def batch(ctx, P, n=130):
        S = P * (P + 1)
        src = rng.normal(size=(n, S))
        p = np.full(n, P, np.uint32)
        return src, lambda: run_device(ctx, "m2l", prec, src, np.zeros((n, S)), p, p, np.tile([2.5, 1.0, 0.5], (n, 1)))

    _, high = batch(native.Context(16, "f64"), 16)
    _, low = batch(native.Context(3, "f64"), 3)
    first = high()
    low()
    assert np.array_equal(high(), first)
