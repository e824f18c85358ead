"""Bloom at the sizes where its passes change form, against the oracle: image sides around the outputs a thread, a
warp and a block take, kernels wider than the image, kernels that do not fit a block's shared memory, and
pixels that are not finite inside and outside the taps whose weights are not zero.  Bars as in
test_post_gpu.py (1e-5 relative for the bloomed image, 1 LSB for the bytes)."""
import numpy as np
import pytest

from test_post_gpu import _check

pytestmark = pytest.mark.gpu


def _image(h, w, seed):
    g = np.random.default_rng(seed)
    img = g.exponential(0.6, (h, w, 4)).astype(np.float32)
    img[g.random((h, w)) < 0.05] = 17.0
    img[..., 3] = 1
    return img


@pytest.mark.parametrize("w,h,radius", [(1, 1, 5.0), (1, 97, 9.0), (8, 95, 0.4), (9, 96, 3.0), (31, 13, 9.0), (33, 12, 60.0),
                                        (287, 11, 1.0), (289, 25, 2.0), (1152, 47, 0.7), (1153, 49, 0.7), (2400, 3, 600.0),
                                        (4617, 2, 1.3), (20000, 2, 0.5)])
def test_sizes(R, O, gpu_ctx, w, h, radius):
    for threshold in (0.0, 1.0):
        _check(R, O, gpu_ctx, _image(h, w, w + h), radius, threshold, 0.3, 0.5)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("channel", [0, 1, 2])
def test_values_that_are_not_finite_spread_over_the_whole_kernel(R, O, gpu_ctx, value, channel):
    """Radius 2 at 700 x 300: 42 and 18 taps a side, 30 of them not zero in x; the pixel reaches outputs
    through zero weights too (0 * inf is NaN), and outputs beyond the kernel stay finite."""
    img = _image(300, 700, 3)
    img[150, 350, channel] = value
    _, comb = _check(R, O, gpu_ctx, img, 2.0, 0.5, 0.3, 0.0)
    assert np.isfinite(comb[:100]).all() and np.isfinite(comb[150, :300]).all()
    if not value < 0:   # -inf falls below the threshold
        assert np.isnan(comb[150, 350 - 40, channel])
