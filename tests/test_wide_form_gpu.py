"""Casts of few rays (eight lanes per ray, and above those cooperative with spread chunks) against the grid form, bit for bit (any hit: the same hit or miss): ray
counts around the ends of a warp's and a block's groups, where two rays per warp become four, and where the
cooperative form takes over and stops spreading; flat and two-level scenes; rays equal in t to several triangles."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def _rays(R, n, seed):
    g = np.random.default_rng(seed)
    rays = np.zeros(n, R.RAY_DTYPE)
    rays["org"] = g.uniform(-1.3, 1.3, (n, 3))
    rays["dir"] = g.standard_normal((n, 3))
    rays["dir"][::9, 1] = 0.0
    rays["tmax"] = 1e4
    rays["tmin"][::5] = 0.05
    rays["tmax"][::13] = 0.3
    return rays


def _check(R, scene, rays):
    ctx = scene.ctx
    got = R.raycast(ctx, scene, rays), R.raycast(ctx, scene, rays, R.RAY_ANY)
    try:
        ctx.set_tuning(refill=R.REFILL_GRID)
        want = R.raycast(ctx, scene, rays), R.raycast(ctx, scene, rays, R.RAY_ANY)
    finally:
        ctx.set_tuning(refill=0)
    assert got[0].tobytes() == want[0].tobytes()
    assert np.array_equal(got[1]["prim"] != R.MISS, want[1]["prim"] != R.MISS)
    return got[0]


@pytest.fixture(scope="module")
def built(R, gpu_ctx):
    flat, _, _ = scenes.sphere_scene(R, gpu_ctx, 5)
    two = scenes.instanced_field(R).to_product(R, gpu_ctx, accel=R.ACCEL_TWO_LEVEL)
    yield flat, two
    flat.close()
    two.close()


@pytest.mark.parametrize("per_sm,n", [(0, 1), (0, 2), (0, 3), (0, 7), (0, 8), (0, 9), (64, -1), (64, 0), (64, 1), (64, 3), (192, 0),
                                      (192, 1), (256, 0), (256, 1), (600, 0), (600, 1), (1280, -3), (1280, 1)])
def test_counts(R, gpu_ctx, built, per_sm, n):
    n += per_sm * gpu_ctx.sm_count
    for scene in built:
        hits = _check(R, scene, _rays(R, n, n))
        assert n < 100 or (hits["prim"] != R.MISS).any()


def test_equal_t(R, gpu_ctx):
    """Coincident triangles, some in one leaf and some apart: the lowest id wins."""
    g = np.random.default_rng(5)
    v = np.ones((60, 4), np.float32)
    v[:, :3] = np.tile(g.uniform(-1, 1, (15, 3)), (4, 1))
    s = R.Scene(gpu_ctx)
    s.add_object(v, np.arange(60, dtype=np.uint32))
    s.build()
    assert (_check(R, s, _rays(R, 4000, 3))["prim"] != R.MISS).any()
    s.close()


def test_empty(R, gpu_ctx):
    s = R.Scene(gpu_ctx)
    s.define_object(np.zeros((3, 4), np.float32), np.zeros(0, np.uint32))
    s.build()
    hits = _check(R, s, _rays(R, 33, 1))
    assert (hits["prim"] == R.MISS).all()
    s.close()
