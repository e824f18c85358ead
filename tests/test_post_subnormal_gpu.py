"""Blurred values below the smallest normal float are the correctly rounded quotients of the sums, as a plain division
gives them: one-pixel images whose two divisions are followed in exact arithmetic."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ONE = 2 ** 149   # subnormals are multiples of 2^-149


def _rounded(x):
    """x rounded to the nearest float, ties to even (0 <= x < 2^127)."""
    e = -149
    while x >= Fraction(2) ** (e + 24):
        e += 1
    return round(x / Fraction(2) ** e) * Fraction(2) ** e


def _exact(f):
    return Fraction(float(f))


def _blurred(R, ctx, value, radius, scale):
    """Blurred value of a 1 x 1 image, times 2^scale (a power of two large enough to hide the image itself)."""
    img = np.float32([[[value, value, value, 1.0]]])
    _, comb = R.postprocess(ctx, img, radius, 0.0, 2.0 ** scale, 0.0, want_combined=True)
    return _exact(comb[0, 0, 0])


@pytest.mark.parametrize("radius", [17.0, 50.0, 100.0])
def test_subnormal_quotients(R, gpu_ctx, radius):
    """Radius 17, 50, 100: kernels of 3, 5 and 7 taps, of which the image has the middle one, whose weight is 1."""
    k = int(np.float32(radius) / np.float32(100) * np.float32(3) + np.float32(0.5))
    near = [np.exp(-i * i / (2.0 * radius * radius)) for i in range(1, k + 1)]
    # the sum of weights is one of the floats around the exact sum: the ones that explain ordinary quotients
    middle = np.float32(1 + 2 * sum(near))
    sums = [np.float32(middle + d * np.spacing(middle)) for d in range(-8, 9)]
    g = np.random.default_rng(int(radius))
    for v in g.uniform(1, 2, 40).astype(np.float32):
        got = _blurred(R, gpu_ctx, v * np.float32(2.0 ** -100), radius, 60)
        want = {float(s): _rounded(_rounded(_exact(v) / _exact(s)) / _exact(s)) * Fraction(2) ** -40 for s in sums}
        sums = [s for s in sums if want[float(s)] == got]
    assert len(sums) == 1
    s = _exact(sums[0])
    wrong = []
    for shift in (126, 127, 128, 130, 140, 147):
        for v in g.uniform(1, 2, 120).astype(np.float32):
            p = np.float32(np.float64(v) * 2.0 ** -(shift - 2))   # quotients from 2^-shift up
            once = _rounded(_exact(p) / s)
            want = _rounded(once / s)
            got = _blurred(R, gpu_ctx, p, radius, 0) - _exact(p)   # image + blurred value, exact where both are so small
            if abs(want) * 2 ** 126 <= 1 and _exact(p) < Fraction(2) ** -123 and got != _rounded(_exact(p) + want) - _exact(p):
                wrong.append((float(p), float(got * ONE), float(want * ONE)))
    assert not wrong, wrong[:4]
