"""The cooperative ray casts against the grid form, bit for bit (any hit: the same hit or miss), where the warps'
lists change form: ray counts around a warp's chunk and a block, every refill threshold, two-level scenes
(instances with and without triangles, several per top-level leaf, one alone), stacks deeper than their
shared part, and hits whose refinement has no determinant."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def _random_rays(R, n, seed, spread=1.2):
    g = np.random.default_rng(seed)
    rays = np.zeros(n, R.RAY_DTYPE)
    rays["org"] = g.uniform(-spread, spread, (n, 3))
    d = g.standard_normal((n, 3)).astype(np.float32)
    d[: n // 16, 1:] = 0.0
    d[n // 16: n // 8, 2] = -0.0
    rays["dir"] = d
    rays["tmax"] = 1e4
    rays["tmin"][::7] = 0.05
    rays["tmax"][::11] = 0.4
    return rays


def _same(R, scene, rays, refills=(1, 8, 32)):
    ctx = scene.ctx
    try:
        ctx.set_tuning(refill=R.REFILL_GRID)
        closest = R.raycast(ctx, scene, rays).view(np.uint32)
        hit = R.raycast(ctx, scene, rays, R.RAY_ANY)["prim"] != R.MISS
        for refill in refills:
            ctx.set_tuning(refill=refill)
            assert np.array_equal(R.raycast(ctx, scene, rays).view(np.uint32), closest), refill
            assert np.array_equal(R.raycast(ctx, scene, rays, R.RAY_ANY)["prim"] != R.MISS, hit), refill
    finally:
        ctx.set_tuning(refill=0)
    return closest.reshape(-1, 4)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129, 4097])
def test_counts(R, gpu_ctx, n):
    flat, _, _ = scenes.sphere_scene(R, gpu_ctx, 4)
    _same(R, flat, _random_rays(R, n, n))
    two = scenes.instanced_field(R).to_product(R, gpu_ctx, accel=R.ACCEL_TWO_LEVEL)
    assert two.stats()["two_level"] == 1
    _same(R, two, _random_rays(R, n, n + 1))


@pytest.mark.parametrize("instances", [1, 2, 3, 5, 64])
def test_two_level_scenes(R, gpu_ctx, instances):
    g = np.random.default_rng(instances)
    s = R.Scene(gpu_ctx)
    s.set_accel(R.ACCEL_TWO_LEVEL)
    v, i, _ = R.icosphere(3, 0.1, 2)
    ball = s.define_object(v, i)
    empty = s.define_object(np.zeros((3, 4), np.float32), np.zeros(0, np.uint32))
    for k in range(instances):
        m = scenes.translate(*g.uniform(-0.5, 0.5, 3)) @ scenes.rotate_y(40.0 * k) @ scenes.scale(*g.uniform(0.1, 0.6, 3))
        s.add_instance(ball, m)
        if k % 2:
            s.add_instance(empty, scenes.translate(*g.uniform(-0.5, 0.5, 3)))
    s.build()
    hits = _same(R, s, _random_rays(R, 20_000, instances))
    assert 0.02 < (hits[:, 0] != R.MISS).mean() < 1.0


def test_deep_stacks(R, gpu_ctx):
    """Overlapping shells of triangles: a ray holds pending children on every level of a deep tree."""
    g = np.random.default_rng(5)
    n = 60_000
    c = (g.standard_normal((n, 1, 3)) * np.exp(g.uniform(-9, 0, (n, 1, 1)))).astype(np.float32)
    t = c + g.standard_normal((n, 3, 3)).astype(np.float32) * np.linalg.norm(c, axis=2, keepdims=True) * 0.3
    s = R.Scene(gpu_ctx)
    s.add_object(t.reshape(-1, 3).astype(np.float32), np.arange(3 * n, dtype=np.uint32))
    s.build()
    assert s.stats()["max_depth"] > 6
    _same(R, s, _random_rays(R, 20_000, 3, 0.2), refills=(8,))


def test_hits_without_a_determinant(R, gpu_ctx):
    """A triangle of 1e-15 hit along a direction of 1e-20: the refinement's determinant underflows to zero and the
    test's own t, u, v are reported."""
    s = R.Scene(gpu_ctx)
    s.add_object(np.float32([[-1e-15, -1e-15, 0], [1e-15, -1e-15, 0], [0, 1e-15, 0]]), np.uint32([0, 1, 2]))
    s.build()
    rays = np.zeros(40, R.RAY_DTYPE)
    rays["org"][:, 0] = np.linspace(-6e-16, 6e-16, 40)
    rays["org"][:, 2] = -1e-14
    rays["dir"][:, 2] = 1e-20
    rays["tmax"] = 1e30
    hits = _same(R, s, rays)
    assert (hits[:, 0] == 0).sum() > 10
