"""Images with pixels that are not finite against the oracle: kernels whose taps all have weight and kernels that end in
taps of weight zero, wider and narrower than a block's rows, with one such pixel, some, and whole rows and
columns of them.  Bars as in test_post_gpu.py."""
import numpy as np
import pytest

from test_post_gpu import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,radius", [(1, 1, 9.0), (13, 100, 9.0), (97, 61, 0.4), (130, 49, 3.0), (200, 300, 2.0), (33, 500, 1.5),
                                        (700, 97, 4.0), (40, 30, 200.0)])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("many", ["one", "some", "lines"])
def test_not_finite(R, O, gpu_ctx, w, h, radius, value, many):
    g = np.random.default_rng(w + h)
    img = g.exponential(0.6, (h, w, 4)).astype(np.float32)
    img[..., 3] = 1
    if many == "one":
        img[h // 2, w // 3, g.integers(3)] = value
    elif many == "some":
        for c in range(3):
            img[g.random((h, w)) < 0.004, c] = value
        img[h - 1, w - 1, 1] = -value
    else:
        img[h // 3, :, 0] = value
        img[:, w // 2, 2] = value
    _check(R, O, gpu_ctx, img, radius, -np.inf if value < 0 else 0.4, 0.3, 0.5)
