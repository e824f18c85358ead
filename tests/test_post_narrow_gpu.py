"""Narrow images, whose rows the blur takes several to a block, against the oracle: widths up to the line where a block
takes one row again, heights around a block's rows, with and without a NaN.  Bars as in test_post_gpu.py."""
import numpy as np
import pytest

from test_post_gpu import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 383), (1, 385), (1, 2000), (2, 192), (7, 55), (30, 12), (30, 13), (31, 1), (31, 25), (32, 24)])
@pytest.mark.parametrize("radius", [0.3, 9.0])
def test_narrow(R, O, gpu_ctx, w, h, radius):
    g = np.random.default_rng(w + h)
    img = g.exponential(0.6, (h, w, 4)).astype(np.float32)
    img[..., 3] = 1
    _check(R, O, gpu_ctx, img, radius, 0.4, 0.3, 0.5)
    img[h // 2, w - 1, 1] = np.nan
    _check(R, O, gpu_ctx, img, radius, 0.4, 0.3, 0.5)
