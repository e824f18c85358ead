"""The roundings of the post-process's sums of three products (luminance, tone map) and what they decide, in exact
arithmetic: which product of a sum is rounded by itself is part of the image's bytes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

f32, wide = np.float32, np.longdouble
N = 700


def _fma(a, b, c):
    return (wide(1) * a * wide(f32(b) if np.isscalar(b) else b) + (wide(f32(c)) if np.isscalar(c) else c)).astype(f32)


def _sum3(a, ka, b, kb, c, kc):
    return _fma(c, kc, _fma(a, ka, (b * f32(kb)).astype(f32)))


def _fit(x):
    return _fma(x, (x + f32(0.0245786)).astype(f32), -0.000090537) / _fma(x, _fma(x, 0.983729, 0.4329510), 0.238081)


def _image(seed, blue):
    g = np.random.default_rng(seed)
    img = g.gamma(0.8, 1.2, (N, N, 4)).astype(f32)
    img[..., 2] *= f32(blue)
    img[..., 3] = 1
    return img


needs_quad = pytest.mark.skipif(np.finfo(wide).nmant < 100, reason="needs 113-bit arithmetic for exact products and sums")


@needs_quad
@pytest.mark.parametrize("blue", [1.0, 0.1, 0.0])
def test_tone_map_bytes(R, gpu_ctx, blue):
    img = _image(int(10 * blue), blue)
    out, _ = R.postprocess(gpu_ctx, img, 1e-6, 1e30, 0.0, 0.0)   # no bloom: every pixel is below the threshold
    r, g, b = (img[..., k] for k in range(3))
    x = _fit(_sum3(r, 0.59719, g, 0.35458, b, 0.04823))
    y = _fit(_sum3(r, 0.07600, g, 0.90834, b, 0.01566))
    z = _fit(_sum3(r, 0.02840, g, 0.13383, b, 0.83777))
    want = [_sum3(x, 1.60475, y, -0.53108, z, -0.07367), _sum3(y, 1.10813, x, -0.10208, z, -0.00605),
            _sum3(x, -0.00327, y, -0.07276, z, 1.07602)]
    for k in range(3):
        v = np.minimum(np.maximum(want[k], f32(0)), f32(1)) * f32(255)
        assert np.array_equal(out[..., k], np.rint(v).astype(np.uint8)), k


@needs_quad
@pytest.mark.parametrize("bad", [False, True])
def test_luminance_at_the_threshold(R, gpu_ctx, bad):
    """Pixels whose luminance is the threshold to within roundings, each its own kernel (radius 1e-6), also where a NaN in
    the image takes the blocks through their other passes."""
    base = np.random.default_rng(3).random((N, N, 3)).astype(f32) + f32(0.01)
    p = base / (base @ f32([0.299, 0.587, 0.114]))[..., None]
    img = np.concatenate([p, np.ones((N, N, 1), f32)], -1).astype(f32)
    if bad:
        img[::7, ::31, 1] = np.nan
    _, comb = R.postprocess(gpu_ctx, img, 1e-6, 1.0, 1.0, 0.0, want_combined=True)
    lum = _sum3(img[..., 0], 0.299, img[..., 1], 0.587, img[..., 2], 0.114)
    want = img[..., 0] * np.where(lum < 1, f32(1), f32(2))
    assert 0.1 < (lum < 1).mean() < 0.9
    assert np.array_equal(comb[..., 0], want)
