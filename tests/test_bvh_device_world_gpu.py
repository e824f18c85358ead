"""Flat scenes built on the device, whose world-space triangles are formed there, against the host build: the same
nodes and triangle records byte for byte and the same hits, with one and many instances, triangle counts
around a block's, models defined after others, per-face materials and an instance without triangles; and
a build that fails leaves no device memory behind."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def _mesh(tris, seed):
    g = np.random.default_rng(seed)
    v = np.ones((3 * tris, 4), np.float32)
    v[:, :3] = (g.uniform(-1, 1, (tris, 1, 3)) + 0.1 * g.standard_normal((tris, 3, 3))).reshape(-1, 3)
    return v, g.permutation(3 * tris).astype(np.uint32)


def _scene(R, ctx, counts, device, per_face=False):
    g = np.random.default_rng(sum(counts) + len(counts))
    s = R.Scene(ctx)
    s.set_accel(R.ACCEL_FLAT)
    s.set_bvh_build(R.BVH_DEVICE if device else R.BVH_HOST, 0)
    ids = [s.define_object(*_mesh(n, n)) for n in counts]
    for k, o in enumerate(ids):
        m = scenes.translate(*g.uniform(-2, 2, 3)) @ scenes.rotate_y(37.0 * k) @ scenes.scale(*g.uniform(-1.5, 1.5, 3))
        if per_face and counts[k]:
            s.add_instance_per_face(o, m, [R.Material(), R.Material(material_idx=1)], np.arange(counts[k]) % 2)
        else:
            s.add_instance(o, m, R.Material())
    s.build()
    return s


@pytest.mark.parametrize("counts,per_face", [((1,), False), ((2,), True), ((127,), False), ((128,), False), ((129,), True),
                                             ((5, 0, 3), False), ((1000, 1, 300, 0), True), ((64,) * 40, False), ((20000,), False)])
def test_same_as_host(R, gpu_ctx, counts, per_face):
    a, b = (_scene(R, gpu_ctx, counts, d, per_face) for d in (False, True))
    for x, y in zip(a.export_bvh(), b.export_bvh()):
        assert x.tobytes() == y.tobytes()
    for k in ("bounds_min", "bounds_max"):
        assert a.stats()[k] == b.stats()[k]
    g = np.random.default_rng(1)
    rays = np.zeros(3000, R.RAY_DTYPE)
    rays["org"] = g.uniform(-4, 4, (3000, 3))
    rays["dir"] = g.uniform(-2, 2, (3000, 3)) - rays["org"]
    rays["tmax"] = 1e4
    hits = [R.raycast(gpu_ctx, s, rays) for s in (a, b)]
    assert hits[0].tobytes() == hits[1].tobytes()
    # a coherence-ordered cast bins the rays over the scene's bounds
    try:
        gpu_ctx.set_tuning(refill=R.REFILL_GRID, trace_order=1)
        assert R.raycast(gpu_ctx, b, rays).tobytes() == hits[0].tobytes()
    finally:
        gpu_ctx.set_tuning(refill=0, trace_order=0)
    a.close()
    b.close()


def test_failed_build(R, gpu_ctx):
    s = R.Scene(gpu_ctx)
    s.set_bvh_build(R.BVH_DEVICE, 0)
    v, i = _mesh(50, 3)
    v[7, 1] = np.inf
    s.add_object(v, i)
    for _ in range(2):
        with pytest.raises(R.ReinaError, match="non-finite"):
            s.build()
    s.close()
