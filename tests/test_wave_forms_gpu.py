"""The wave engine's forms against the pass-by-pass engine, sample by sample and bit for bit: cooperative and grid
traversal, waves cut for overlap, one scene's or several scenes' jobs, flat and two-level, direct launches
and graphs, only some materials present, and bounces past the ring of per-bounce counters."""
import ctypes as C

import numpy as np
import pytest
import torch

import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(R):
    c = R.Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def built(R, ctx):
    def sphere(level, **mat):
        d = scenes.cornell(R)
        v, i, tbn, ti = scenes.sphere_tbn(level, 0.1, 3, R)
        d.add_instance(d.add_object(v, i, tbn, ti), scenes.translate(0, -0.3, 0.2) @ scenes.scale(0.6, 0.6, 0.6), R.Material(**mat))
        return d.to_product(R, ctx)
    one = dict(specular_tint=(1, 1, 1), sheen_tint=(1, 1, 1))
    return {
        "few_nodes": sphere(2, albedo=(0.7, 0.5, 0.3), interp_normals=True),
        "nodes": sphere(5, material_idx=3, albedo=(0.7, 0.3, 0.2), roughness=0.3, metallic=0.6, **one),
        "metal": sphere(5, material_idx=1, albedo=(0.9, 0.8, 0.6), roughness=0.2),
        "glass": sphere(5, material_idx=2, albedo=(0.8, 0.9, 0.95), ior=1.5, absorption=1.5, roughness=0.05),
        "textured": scenes.textured_room(R).to_product(R, ctx),
        "zoo": scenes.material_zoo(R).to_product(R, ctx),
        "instanced": scenes.instanced_field(R).to_product(R, ctx, accel=R.ACCEL_TWO_LEVEL),
    }


def frame(R, scene, w, h, spp=2, bounces=5, mode=1, **options):
    iv, ip = scenes.cornell_camera(R, w, h)
    pc = R.push_consts(iv, ip, total_emissive_weight=scene.emissive_weight, spp=spp, max_bounces=bounces, focus_dist=3.4)
    return pc, R.render_options(w, h, mode, 7, **options)


def samples(R, ctx, jobs):
    """The jobs' samples and images in one call without counters (one job: reina_render_device)."""
    out = [(torch.zeros((o.height, o.width, 4), device="cuda"),
            torch.zeros((o.height * o.width, pc.samplesPerPixel, 3), device="cuda")) for _, pc, o in jobs]
    if len(jobs) == 1:
        s, pc, o = jobs[0]
        R.render_device(ctx, s, pc, o, out[0][0].data_ptr(), out[0][1].data_ptr())
    else:
        arr = R._jobs_array([R.DeviceRenderJob(s, pc, o, a.data_ptr(), b.data_ptr()) for (s, pc, o), (a, b) in zip(jobs, out)], True)
        assert R._lib.reina_render_batch_device(ctx.handle, arr, len(jobs), C.c_void_p(0), None) == R.REINA_OK
    torch.cuda.synchronize()
    return [tuple(t.cpu().numpy().view(np.uint32) for t in pair) for pair in out]


def forms(R, ctx, jobs):
    """Every form's samples and images: the engine's choice, cooperative by request, with direct launches."""
    try:
        for kw in (dict(), dict(wave_refill=1), dict(wave_refill=8), dict(batch_flags=R.BATCH_NO_GRAPHS),
                   dict(wave_refill=8, batch_flags=R.BATCH_NO_GRAPHS)):
            ctx.set_tuning(**{"wave_refill": R.REFILL_GRID, "batch_flags": 0, **kw})
            yield kw, samples(R, ctx, jobs)
    finally:
        ctx.set_tuning(wave_refill=R.REFILL_GRID, batch_flags=0)


def same(got, want, kw):
    for g, w in zip(got, want):
        for a, b in zip(g, w):
            nan = np.isnan(a.view(np.float32)) & np.isnan(b.view(np.float32))
            assert np.array_equal(a[~nan], b[~nan]), kw


# 61x47: one small wave; 512x512 and 513x511 in the reference's mode: 2^18 paths and one row more or less, where grid-form
# calls begin to be cut; 1024x1024: 2^20, where two-level scenes turn cooperative
@pytest.mark.parametrize("name,w,h,spp,mode", [
    *[(n, 61, 47, 3, m) for n in ("few_nodes", "nodes", "metal", "glass", "textured", "zoo", "instanced") for m in (0, 1)],
    ("few_nodes", 512, 512, 1, 0), ("few_nodes", 511, 512, 2, 0), ("few_nodes", 301, 299, 3, 1), ("instanced", 1024, 1024, 1, 0),
    ("instanced", 1023, 1024, 1, 0), ("nodes", 733, 641, 1, 1)])
def test_forms(R, ctx, built, name, w, h, spp, mode):
    s = built[name]
    want = samples(R, ctx, [(s, *frame(R, s, w, h, spp, mode=mode, pass_by_pass=True))])
    for kw, got in forms(R, ctx, [(s, *frame(R, s, w, h, spp, mode=mode))]):
        same(got, want, kw)


@pytest.mark.parametrize("names", [("few_nodes", "nodes"), ("metal", "instanced", "few_nodes"), ("instanced", "instanced"),
                                   ("glass", "zoo", "textured", "nodes", "metal")])
def test_mixed_jobs(R, ctx, built, names):
    shapes = [(61, 47, 3, 4, 1), (33, 80, 1, 7, 0), (200, 150, 2, 3, 1), (16, 16, 9, 0, 1), (97, 31, 2, 12, 0)]
    jobs, want = [], []
    for k, n in enumerate(names):
        w, h, spp, bounces, mode = shapes[k]
        jobs.append((built[n], *frame(R, built[n], w, h, spp, bounces, mode)))
        want += samples(R, ctx, [(built[n], *frame(R, built[n], w, h, spp, bounces, mode, pass_by_pass=True))])
    for kw, got in forms(R, ctx, jobs):
        same(got, want, kw)


@pytest.mark.parametrize("bounces", [511, 512, 513, 1024, 1025, 1600])
def test_deep_bounces(R, ctx, bounces):
    """A closed metal shell: paths go on to the last bounce, whose counters reuse those of earlier ones."""
    d = scenes.SceneDesc()
    v, i, _ = R.icosphere(2, 0.1, 5)
    d.add_instance(d.add_object(v, i), scenes.scale(40, 40, 40), R.Material(material_idx=1, albedo=(1, 1, 1), roughness=0.3,
                                                                             emission=(0.01, 0.02, 0.03)))
    s = d.to_product(R, ctx)
    want = samples(R, ctx, [(s, *frame(R, s, 9, 7, 2, bounces, pass_by_pass=True))])
    assert want[0][1].view(np.float32).max() > 0
    for kw, got in forms(R, ctx, [(s, *frame(R, s, 9, 7, 2, bounces))]):
        same(got, want, kw)
    s.close()


@pytest.mark.parametrize("level", [0, 3, 6])
def test_exported_triangles_hold_no_tags(R, ctx, level):
    """The device copy of a flat scene's triangle records carries instance data in its spare words, the exported does not."""
    s, _, _ = scenes.sphere_scene(R, ctx, level)
    _, tris = s.export_bvh()
    words = tris.view(np.uint32).reshape(-1, 12)
    assert not words[:, [7, 11]].any()


@pytest.mark.parametrize("name,per_sm", [("few_nodes", 96), ("instanced", 192), ("nodes", 352)])
@pytest.mark.parametrize("extra", [0, 1])
def test_few_paths(R, ctx, built, name, per_sm, extra):
    """As many paths as are traced with eight lanes per ray, and one column more."""
    w = per_sm + extra
    s = built[name]
    want = samples(R, ctx, [(s, *frame(R, s, w, ctx.sm_count, 1, mode=0, pass_by_pass=True))])
    for kw, got in forms(R, ctx, [(s, *frame(R, s, w, ctx.sm_count, 1, mode=0))]):
        same(got, want, kw)


@pytest.mark.parametrize("w,h,spp", [(520, 511, 3), (601, 600, 4), (512, 515, 2), (1, 262145, 2)])
def test_carried_samples_in_cut_waves(R, ctx, built, w, h, spp):
    """The reference's mode, whose samples of a pixel start from the state the last one left, in waves cut to overlap."""
    s = built["few_nodes"]
    want = samples(R, ctx, [(s, *frame(R, s, w, h, spp, 4, mode=0, pass_by_pass=True))])
    for kw, got in forms(R, ctx, [(s, *frame(R, s, w, h, spp, 4, mode=0))]):
        same(got, want, kw)
    jobs = [(s, *frame(R, s, w, h, spp, 4, mode=0)), (built["instanced"], *frame(R, built["instanced"], 40, 30, 7, 3, mode=0))]
    want += samples(R, ctx, [(jobs[1][0], *frame(R, jobs[1][0], 40, 30, 7, 3, mode=0, pass_by_pass=True))])
    same(samples(R, ctx, jobs), want, "two jobs")
