"""Timed workloads of the trace path, through the calls a program makes.

Five kinds of work: ray casts (device or page-locked host buffers, closest or any hit, flat or instanced
scenes), frames (both integrator modes, one-shot and progressive), batched frames, the post-process of a
rendered image, and building a scene with the device BVH builder.  The mesh of every kind is a displaced
geodesic sphere of 20 * frequency^2 triangles, the synthetic geometry this repository uses throughout.

listed() names fixed cases, draw() gives more of the same ranges; prepare() makes what a program holds
before the call (scene, rays, images), run() is one call and its outputs, work() the bytes and operations
it cannot do without and exact() the outputs in 64 bits where they have such a value.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), os.pardir, "reina-vk_gb300"))
import reina_gb300 as R  # noqa: E402

T_MAX = 1.0e4
ENV = (0.3, 0.3, 0.35)
EXACT_PAIRS = 3.0e10   # ray-triangle pairs of a brute-force 64-bit cast: about ten seconds

_ctx = None


def _context():
    """The one context a program holds on a GPU."""
    global _ctx
    if _ctx is None:
        _ctx = R.Context(0)
    return _ctx


def _stream():
    return torch.cuda.current_stream().cuda_stream


# ---------------------------------------------------------------------------------------------------
# Cases

def listed():
    return [
        # Picking and visibility probes between frames of an editor: a thousand rays, latency is all.
        dict(name="cast_probe", kind="cast", frequency=64, side=24, random=424, any=False, where="device", instances=0),
        # An ordinary ray query of a mid-size mesh, odd counts.
        dict(name="cast_mid", kind="cast", frequency=64, side=391, random=150_001, any=False, where="device", instances=0),
        # The benchmark's own step: 1.3M triangles, 1024 x 1024 camera rays and as many random ones.
        dict(name="cast_large", kind="cast", frequency=256, side=1024, random=1 << 20, any=False, where="device",
             instances=0),
        # The same rays as visibility (shadow, ambient occlusion) queries.
        dict(name="cast_large_any", kind="cast", frequency=256, side=1024, random=1 << 20, any=True, where="device",
             instances=0),
        # The same step from and to page-locked host memory: the benchmark's end-to-end call.
        dict(name="cast_large_host", kind="cast", frequency=256, side=1024, random=1 << 20, any=False, where="host",
             instances=0),
        # An instanced scene (two-level structure): 256 copies of a 20,480-triangle model.
        dict(name="cast_instanced", kind="cast", frequency=32, side=1024, random=1 << 20, any=False, where="device",
             instances=256),
        # A preview frame of a small room, the benchmark's: 256 x 256, 16 samples, 8 bounces, NEE + MIS.
        dict(name="frame_room", kind="frame", scene="room", frequency=0, width=256, height=256, spp=16, bounces=8,
             nee=True, progressive=False),
        # The application's loop: its 1080 x 1350 window, one sample a frame blended into the image, every
        # material and textures, the integrator as the application ships it.
        dict(name="frame_window", kind="frame", scene="zoo", frequency=24, width=1080, height=1350, spp=1, bounces=9,
             nee=False, progressive=True),
        # A quarter of the benchmark's large frame: 1920 x 1080, 12 bounces, 1.3M triangles.
        dict(name="frame_large", kind="frame", scene="sphere", frequency=256, width=1920, height=1080, spp=16,
             bounces=12, nee=True, progressive=False),
        # A queue of small jobs of several scenes, sizes and depths rendered together.
        dict(name="batch", kind="batch", jobs=12, frequency=90, side=320, spp=12, bounces=10),
        # Bloom and tone map of a full-HD image with the application's default settings.
        dict(name="post_hd", kind="post", width=1920, height=1080, radius=5.0, threshold=1.0, combined=True),
        # Loading a mesh into a scene: assembly, device BVH build, upload.
        dict(name="build_mid", kind="build", frequency=128, bins=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cast", "cast", "cast", "frame", "frame", "batch", "post", "build"])
    if kind == "cast":
        inst = rng.choice([0, 0, 0, _log(rng, 8, 256)])
        return dict(kind="cast", frequency=_log(rng, 4, 32) if inst else _log(rng, 6, 256), side=_log(rng, 8, 1024),
                    random=_log(rng, 64, 1 << 20), any=rng.random() < 0.3, where=rng.choice(["device", "device", "host"]),
                    instances=inst)
    if kind == "frame":
        scene = rng.choice(["room", "zoo", "sphere", "field"])
        return dict(kind="frame", scene=scene, frequency=_log(rng, 8, 160) if scene == "sphere" else _log(rng, 6, 32),
                    width=_log(rng, 61, 1920), height=_log(rng, 47, 1080), spp=_log(rng, 1, 16),
                    bounces=rng.randint(3, 12), nee=rng.random() < 0.7, progressive=rng.random() < 0.3)
    if kind == "batch":
        return dict(kind="batch", jobs=rng.randint(2, 12), frequency=_log(rng, 8, 90), side=_log(rng, 65, 320),
                    spp=_log(rng, 1, 12), bounces=rng.randint(4, 10))
    if kind == "post":
        return dict(kind="post", width=_log(rng, 33, 1920), height=_log(rng, 21, 1080),
                    radius=round(rng.uniform(0.3, 9.0), 2), threshold=round(rng.uniform(0.0, 2.0), 2),
                    combined=rng.random() < 0.5)
    return dict(kind="build", frequency=_log(rng, 4, 128), bins=rng.choice([0, 16]))


# ---------------------------------------------------------------------------------------------------
# Geometry

def _sphere(frequency, seed):
    """A displaced geodesic sphere with tangent frames: vertices (N, 4), indices, TBNs (N, 9)."""
    v, i, n = R.geodesic(frequency, 0.1, seed)
    up = np.where(np.abs(n[:, 1:2]) > 0.99, np.float32([[1, 0, 0]]), np.float32([[0, 1, 0]]))
    t = np.cross(up, n)
    t /= np.linalg.norm(t, axis=1, keepdims=True)
    return v, i, np.concatenate([t, np.cross(n, t), n], axis=1).astype(np.float32)


def _quad(corner, e1, e2):
    c, a, b = (np.asarray(x, np.float32) for x in (corner, e1, e2))
    return np.stack([c, c + a, c + a + b, c + b]), np.array([0, 1, 2, 0, 2, 3], np.uint32)


def _cube():
    v = np.array([[x, y, z] for z in (-.5, .5) for y in (-.5, .5) for x in (-.5, .5)], np.float32)
    i = np.array([0, 2, 3, 0, 3, 1, 4, 5, 7, 4, 7, 6, 0, 4, 6, 0, 6, 2, 1, 3, 7, 1, 7, 5, 0, 1, 5, 0, 5, 4, 2, 6, 7, 2,
                  7, 3], np.uint32)
    return v, i


def _move(x, y, z, s=1.0, turn=0.0, tall=1.0):
    """Scale by s (and tall in y), turn about y (radians), translate."""
    c, k = math.cos(turn), math.sin(turn)
    return np.array([[c * s, 0, k * s, x], [0, s * tall, 0, y], [-k * s, 0, c * s, z], [0, 0, 0, 1]], np.float32)


def _instances(n, seed):
    """n rotated and scaled copies spread over [-1, 1]^3."""
    g = np.random.default_rng(seed)
    out = []
    for _ in range(n):
        q, r = np.linalg.qr(g.standard_normal((3, 3)))
        q *= np.sign(np.diag(r))
        m = np.eye(4)
        m[:3, :3] = q @ np.diag(g.uniform(0.04, 0.16, 3))
        m[:3, 3] = g.uniform(-0.9, 0.9, 3)
        out.append(m.astype(np.float32))
    return out


def _palette(seed, count=256):
    """Disney materials, one in five of them glass."""
    g = np.random.default_rng(seed).random((count, 12))
    one = (1.0, 1.0, 1.0)
    return [R.Material(material_idx=2, albedo=tuple(0.6 + 0.4 * r[:3]), ior=1.5, absorption=2.0 * r[3]) if r[11] < 0.2 else
            R.Material(material_idx=3, albedo=tuple(r[:3]), metallic=r[3], roughness=0.05 + 0.95 * r[4],
                       clearcoat=r[6], sheen=r[7], clearcoat_gloss=r[8], sheen_tint=one, specular_tint=one)
            for r in g]


def _sphere_scene(frequency, seed):
    """The sphere with per-face materials over a ground plane, under a quad light."""
    s = R.Scene(_context())
    s.set_bvh_build(R.BVH_DEVICE)
    v, i, t = _sphere(frequency, seed)
    o = s.define_object(v, i, tbns=t, tbn_indices=i)
    faces = np.random.default_rng(seed).integers(0, 256, i.size // 3).astype(np.uint32)
    s.add_instance_per_face(o, None, _palette(seed), faces)
    s.add_object(*_quad((-10, -1.2, 10), (20, 0, 0), (0, 0, -20)), material=R.Material(albedo=(0.5, 0.5, 0.5)))
    s.add_object(*_quad((-0.75, 2.5, -0.75), (1.5, 0, 0), (0, 0, 1.5)),
                 material=R.Material(albedo=(0.9, 0.9, 0.9), emission=(17.0, 12.0, 4.0), cull_backface=True))
    s.build(require_emissive=True)
    return s


def _room_scene(scene, frequency, seed):
    """A box room lit by a ceiling quad: with two boxes ("room"), with spheres of every material and
    textured surfaces ("zoo"), or with many instances of one sphere ("field", a two-level structure)."""
    g = np.random.default_rng(seed)
    s = R.Scene(_context())
    grey, M = (0.73, 0.73, 0.73), R.Material
    albedo = normals = -1
    uv = np.array([[0, 0], [3, 0], [3, 3], [0, 3]], np.float32)
    if scene == "zoo":
        tex = np.full((64, 64, 4), 255, np.uint8)
        tex[..., :3] = np.kron(g.integers(60, 256, (8, 8, 3)), np.ones((8, 8, 1)))
        albedo = s.define_texture_rgba8(tex)
        n = np.concatenate([g.uniform(-0.2, 0.2, (64, 64, 2)), np.ones((64, 64, 1))], -1)
        n = n / np.linalg.norm(n, axis=-1, keepdims=True)
        normals = s.define_texture_rgba8(np.concatenate([np.round((n * 0.5 + 0.5) * 255), np.full((64, 64, 1), 255)],
                                                        -1).astype(np.uint8))
    walls = [((-1, -1, 1), (2, 0, 0), (0, 0, -2), grey), ((-1, 1, -1), (2, 0, 0), (0, 0, 2), grey),
             ((-1, -1, -1), (2, 0, 0), (0, 2, 0), grey), ((-1, -1, 1), (0, 0, -2), (0, 2, 0), (0.65, 0.05, 0.05)),
             ((1, -1, -1), (0, 0, 2), (0, 2, 0), (0.12, 0.45, 0.15))]
    for k, (c, a, b, col) in enumerate(walls):
        v, i = _quad(c, a, b)
        t, bt = np.asarray(a, np.float32) / 2, np.asarray(b, np.float32) / 2
        tbn = np.tile(np.concatenate([t, bt, np.cross(t, bt)]), (4, 1)).astype(np.float32)
        s.add_object(v, i, material=M(albedo=col, texture_id=albedo if k == 0 else -1,
                                      normal_map_id=normals if k in (0, 2) else -1),
                     tbns=tbn, tbn_indices=i, tex_coords=uv, tex_indices=i)
    if scene == "room":
        box = s.define_object(*_cube())
        s.add_instance(box, _move(-0.35, -0.4, -0.3, 0.6, math.radians(15 + 5 * g.random()), 2.0), M(albedo=grey))
        s.add_instance(box, _move(0.35, -0.7, 0.35, 0.6, -math.radians(15 + 5 * g.random())), M(albedo=grey))
    else:
        v, i, t = _sphere(frequency, seed)
        ball = s.define_object(v, i, tbns=t, tbn_indices=i)
        one = dict(specular_tint=(1, 1, 1), sheen_tint=(1, 1, 1))
        mats = [M(material_idx=1, albedo=(0.9, 0.8, 0.6), roughness=0.2),
                M(material_idx=2, albedo=(0.8, 0.9, 0.95), absorption=1.5, roughness=0.05, interp_normals=True),
                M(material_idx=3, albedo=(0.7, 0.3, 0.2), roughness=0.6, subsurface=0.4, sheen=0.8, **one),
                M(material_idx=3, albedo=(0.95, 0.75, 0.3), metallic=0.9, roughness=0.3, anisotropic=0.5, **one),
                M(material_idx=3, albedo=(0.2, 0.4, 0.8), clearcoat=1.0, clearcoat_gloss=0.7, roughness=0.4, **one),
                M(material_idx=3, albedo=(0.9, 0.95, 0.9), specular_transmission=0.8, ior=1.45, roughness=0.15, **one)]
        if scene == "zoo":
            for k, m in enumerate(mats):
                s.add_instance(ball, _move(-0.6 + 0.6 * (k % 3), -0.75 + 1.0 * (k // 3), 0.1 + 0.2 * g.random(), 0.22,
                                           g.random()), m)
        else:
            for k, m in enumerate(_instances(64, seed)):
                s.add_instance(ball, m, mats[k % 6])
    s.add_object(*_quad((-0.25, 0.999, -0.2), (0.5, 0, 0), (0, 0, 0.4)),
                 material=M(albedo=(0.78, 0.78, 0.78), emission=(17.0, 12.0, 4.0), cull_backface=True))
    s.build(require_emissive=True)
    return s


# ---------------------------------------------------------------------------------------------------
# prepare

def _rays(case, seed, lo, hi):
    """side^2 camera rays from a point three units away, then random rays in the box expanded 1.5 times."""
    a = np.random.default_rng(seed).uniform(-0.6, 0.6, 2)
    eye = 3.0 * np.array([math.sin(a[0]) * math.cos(a[1]), math.sin(a[1]), math.cos(a[0]) * math.cos(a[1])])
    c, h = (lo + hi) / 2, (hi - lo) / 2 * 1.5
    return R.raycast_rays(case["side"], case["side"], eye, (0.0, 0.0, 0.0), 45.0, case["random"], c - h, c + h, seed=seed)


def _prepare_cast(case, seed):
    s = R.Scene(_context())
    s.set_bvh_build(R.BVH_DEVICE)
    v, i, _ = R.geodesic(case["frequency"], 0.1, seed)
    o = s.define_object(v, i)
    if case["instances"]:
        s.set_accel(R.ACCEL_TWO_LEVEL)
        for m in _instances(case["instances"], seed):
            s.add_instance(o, m)
    else:
        s.add_instance(o)
    s.build()
    lo, hi = (np.float32([-1.1] * 3), np.float32([1.1] * 3)) if case["instances"] else (v[:, :3].min(0), v[:, :3].max(0))
    rays = _rays(case, seed, lo, hi)
    n = rays.shape[0]
    rays = torch.from_numpy(rays.view(np.float32).reshape(n, 8))
    hits = torch.zeros((n, 4), dtype=torch.int32)
    if case["where"] == "host":
        rays, hits = rays.pin_memory(), hits.pin_memory()
    else:
        rays, hits = rays.cuda(), hits.cuda()
    return dict(kind="cast", scene=s, rays=rays, hits=hits, n=n, host=case["where"] == "host", any=case["any"],
                flags=R.RAY_ANY if case["any"] else R.RAY_CLOSEST,
                out=dict(prim=hits[:, 0], tuv=hits[:, 1:].view(torch.float32)))


def _frame_args(scene, kind, width, height, spp, bounces, nee, seed):
    jitter = np.random.default_rng(seed + 1).uniform(-0.05, 0.05, 2)
    if kind == "sphere":
        pos, front = (jitter[0], 0.4 + jitter[1], 3.6), (0.0, -0.12, -1.0)
    else:
        pos, front = (jitter[0], jitter[1], 3.4), (0.0, 0.0, -1.0)
    iv, ip = R.camera_matrices(pos, front, (0.0, 1.0, 0.0), np.radians(40.0), width / height)
    pc = R.push_consts(iv, ip, total_emissive_weight=scene.emissive_weight, spp=spp, max_bounces=bounces, focus_dist=3.5)
    env = dict(env_mode=R.ENV_CONSTANT, env_color=ENV) if kind == "sphere" else {}
    return pc, R.render_options(width, height, R.MODE_NEE_MIS if nee else R.MODE_REINA, seed & 0x7FFFFFFF, **env)


def _prepare_frame(case, seed):
    if case["scene"] == "sphere":
        scene = _sphere_scene(case["frequency"], seed)
    else:
        scene = _room_scene(case["scene"], case["frequency"], seed)
    w, h = case["width"], case["height"]
    pc, opts = _frame_args(scene, case["scene"], w, h, case["spp"], case["bounces"], case["nee"], seed)
    pc.sampleBatch = seed % 50
    if not case["progressive"]:
        pc.sampleBatch = 0
    g = torch.Generator(device="cuda").manual_seed(seed)
    image = torch.rand((h, w, 4), generator=g, device="cuda")
    return dict(kind="frame", scene=scene, pc=pc, opts=opts, image=image, progressive=case["progressive"])


def _prepare_batch(case, seed):
    g = np.random.default_rng(case["side"] + case["spp"])   # the queue's sizes are the case's, not the seed's
    jobs, images, scenes = [], [], []
    for k in range(case["jobs"]):
        if k < 4:
            scenes.append(_sphere_scene(max(4, case["frequency"] // (k + 1)), seed + k))
        scene = scenes[k % len(scenes)]
        side = max(17, int(case["side"] * g.uniform(0.4, 1.0)))
        pc, opts = _frame_args(scene, "sphere", side, side, max(1, int(case["spp"] * g.uniform(0.4, 1.0))),
                               int(g.integers(3, case["bounces"] + 1)), True, seed + k)
        images.append(torch.zeros((side, side, 4), device="cuda"))
        jobs.append(R.DeviceRenderJob(scene, pc, opts, images[-1].data_ptr()))
    return dict(kind="batch", jobs=jobs, images=images, scenes=scenes)


def _prepare_post(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    w, h = case["width"], case["height"]
    image = torch.empty((h, w, 4), device="cuda").exponential_(2.5, generator=g)
    lit = torch.rand((h // 20 + 1, w // 20 + 1), generator=g, device="cuda") > 0.97   # light sources in view
    image[lit.repeat_interleave(20, 0).repeat_interleave(20, 1)[:h, :w]] = 17.0
    image[..., 3] = 1.0
    rgba = torch.empty((h, w, 4), dtype=torch.uint8, device="cuda")
    out = dict(rgba=rgba)
    if case["combined"]:
        out["combined"] = torch.empty((h, w, 4), device="cuda")
    lib = R.load_library()
    return dict(kind="post", image=image, out=out, width=w, height=h, call=lib.reina_postprocess_device,
                bloom=R.BloomPushConsts(case["radius"], case["threshold"], 0.05), tone=R.TonemappingPushConsts(1.0))


def _prepare_build(case, seed):
    v, i, t = _sphere(case["frequency"], seed)
    tris = _triangles(case["frequency"])
    return dict(kind="build", v=v, i=i, t=t, bins=case["bins"], scene=None,
                nodes=np.zeros((tris // 2 + 8, R.NODE_BYTES), np.uint8))   # room for any mesh's node count


def prepare(case, seed):
    make = dict(cast=_prepare_cast, frame=_prepare_frame, batch=_prepare_batch, post=_prepare_post, build=_prepare_build)
    return make[case["kind"]](case, seed)


# ---------------------------------------------------------------------------------------------------
# run

def run(state):
    kind = state["kind"]
    if kind == "cast":
        if state["host"]:
            R.raycast_into(_context(), state["scene"], state["rays"].data_ptr(), state["n"], state["hits"].data_ptr(),
                           state["flags"])
        else:
            R.raycast_device(_context(), state["scene"], state["rays"].data_ptr(), state["n"], state["hits"].data_ptr(),
                             state["flags"], _stream())
        # which of its occluders an any-hit ray reports is up to the schedule: the answer is hit or miss
        return state["out"]["prim"] != -1 if state["any"] else state["out"]
    if kind == "frame":
        if state["progressive"]:
            state["pc"].sampleBatch += 1
        R.render_device(_context(), state["scene"], state["pc"], state["opts"], state["image"].data_ptr(), 0, _stream())
        return state["image"]
    if kind == "batch":
        R.render_batch_device(_context(), state["jobs"], _stream())
        return state["images"]
    if kind == "post":
        combined = state["out"].get("combined")
        status = state["call"](_context().handle, state["image"].data_ptr(), state["width"], state["height"], state["bloom"],
                               state["tone"], state["out"]["rgba"].data_ptr(),
                               None if combined is None else combined.data_ptr(), _stream())
        if status != R.REINA_OK:
            raise RuntimeError(f"post-process failed: {status}")
        return state["out"]
    if state["scene"] is not None:   # the new mesh replaces the one shown before
        state["scene"].close()
    scene = R.Scene(_context())
    scene.set_bvh_build(R.BVH_DEVICE, state["bins"])
    scene.add_object(state["v"], state["i"], tbns=state["t"], tbn_indices=state["i"])
    scene.build()
    state["scene"] = scene
    nodes, triangles = scene.export_bvh()
    state["nodes"][:len(nodes)] = nodes
    return dict(nodes=state["nodes"], triangles=triangles)


# ---------------------------------------------------------------------------------------------------
# work

def _triangles(frequency):
    return 20 * frequency * frequency


def _scene_bytes(triangles):
    """Traversal data read once: 48 bytes a triangle and an 80-byte node for about nine triangles."""
    return triangles * (48.0 + 80.0 / 9.0)


def _ray_flops(triangles):
    """A ray's box tests (eight boxes of six planes a level, two nodes a level) and its triangle tests."""
    return 2.0 * max(1.0, math.log(max(2.0, triangles), 8)) * 8 * 18 + 4 * 60


def work(case):
    kind = case["kind"]
    if kind == "cast":
        n = case["side"] ** 2 + case["random"]
        t = _triangles(case["frequency"])
        return dict(bytes=48.0 * n + _scene_bytes(t) + 64.0 * case["instances"], flops=n * _ray_flops(t * max(1, case["instances"])))
    if kind in ("frame", "batch"):
        if kind == "frame":
            px, samples = case["width"] * case["height"], case["width"] * case["height"] * case["spp"]
            t = 36 if case["scene"] == "room" else _triangles(case["frequency"])
        else:
            px = case["jobs"] * (0.7 * case["side"]) ** 2
            samples, t = px * 0.7 * case["spp"], _triangles(case["frequency"]) * 1.4
        rays = samples * min(case["bounces"], 4) * (2 if case.get("nee", True) else 1)
        return dict(bytes=px * (32.0 if case.get("progressive") else 16.0) + _scene_bytes(t), flops=rays * (_ray_flops(t) + 500.0))
    if kind == "post":
        px = case["width"] * case["height"]
        taps = sum(min(2 * int(side * case["radius"] / 100 * 3 + 0.5) + 1, 2 * int(14.4 * case["radius"]) + 1)
                   for side in (case["width"], case["height"]))   # taps whose weight is not zero in float
        return dict(bytes=px * (16.0 + 4.0 + (16.0 if case["combined"] else 0.0)), flops=px * (6.0 * taps + 60.0))
    t = _triangles(case["frequency"])
    return dict(bytes=t * (6.0 + 36 + 12 + 48) + t * 80.0 / 9, flops=t * 17.0 * 60)


# ---------------------------------------------------------------------------------------------------
# exact

def _exact_cast(case, seed):
    """Brute force in 64 bits: the closest triangle of every ray by Moller and Trumbore's test."""
    n, t = case["side"] ** 2 + case["random"], _triangles(case["frequency"]) * max(1, case["instances"])
    if case["any"] or n * t > EXACT_PAIRS:
        return None
    v, i, _ = R.geodesic(case["frequency"], 0.1, seed)
    tri = v[i.reshape(-1, 3)][:, :, :3].astype(np.float64)
    lo, hi = v[:, :3].min(0), v[:, :3].max(0)
    if case["instances"]:
        lo, hi = np.float32([-1.1] * 3), np.float32([1.1] * 3)
        ms = [m.astype(np.float64) for m in _instances(case["instances"], seed)]
        tri = np.concatenate([tri @ m[:3, :3].T + m[:3, 3] for m in ms])
    rays = _rays(case, seed, lo, hi).view(np.float32).reshape(n, 8)
    rays = torch.from_numpy(rays).cuda().double()
    tri = torch.from_numpy(tri).cuda()
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    normal = torch.linalg.cross(e1, e2)
    # with m = o x d: det = -d.n, u det = d.(a x e2) + m.e2, v det = -(d.(a x e1) + m.e1), t det = (o - a).n
    lhs_u = torch.cat([torch.linalg.cross(a, e2), e2], 1).T.contiguous()
    lhs_v = torch.cat([-torch.linalg.cross(a, e1), -e1], 1).T.contiguous()
    lhs_t = torch.cat([normal, -(a * normal).sum(1, keepdim=True)], 1).T.contiguous()
    out = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    step = max(1, int(2.0e8 // t))
    for at in range(0, n, step):
        o, d = rays[at:at + step, :3], rays[at:at + step, 4:7]
        od = torch.cat([d, torch.linalg.cross(o, d)], 1)
        det = -(d @ normal.T)
        u = torch.div(od @ lhs_u, det)
        w = torch.div(od @ lhs_v, det)
        dist = torch.div(torch.cat([o, torch.ones_like(o[:, :1])], 1) @ lhs_t, det)
        ok = (u >= 0) & (w >= 0) & (u + w <= 1) & (dist >= 0) & (dist <= T_MAX)
        dist = torch.where(ok, dist, math.inf)
        best, k = dist.min(1)
        hit = best < math.inf
        row = torch.arange(len(k), device="cuda")
        out[at:at + step, 0] = torch.where(hit, best, T_MAX)
        out[at:at + step, 1] = torch.where(hit, u[row, k], 0.0)
        out[at:at + step, 2] = torch.where(hit, w[row, k], 0.0)
    return dict(prim=None, tuv=out)


def _exact_post(case, seed):
    """Bloom as two dense convolutions of the whole kernel."""
    if not case["combined"]:
        return None
    img = _prepare_post(case, seed)["image"].double()[..., :3]
    h, w = img.shape[:2]
    lum = img @ img.new_tensor([0.299, 0.587, 0.114])
    x = torch.where((lum < case["threshold"])[..., None], 0.0, img).permute(2, 0, 1)
    for axis, side in ((2, w), (1, h)):
        k = int(side * case["radius"] / 100 * 3 + 0.5)
        g = torch.exp(-torch.arange(-k, k + 1, device="cuda").double() ** 2 / (2 * case["radius"] ** 2))
        size = 1 << (side + 2 * k).bit_length()
        f = torch.fft.irfft(torch.fft.rfft(x, size, axis) * torch.fft.rfft(g, size).reshape(-1, *([1] * (2 - axis))), size, axis)
        x = f.narrow(axis, k, side) / g.sum()
    out = torch.ones((h, w, 4), dtype=torch.float64, device="cuda")
    out[..., :3] = img + 0.05 * x.permute(1, 2, 0)
    return dict(rgba=None, combined=out)


def exact(case, seed):
    # A path follows comparisons of rounded numbers (roulette, lobe choice, which triangle is nearest), so a
    # frame in 64 bits is a frame of other paths and no value of the same outputs; a build returns bytes.
    if case["kind"] == "cast":
        return _exact_cast(case, seed)
    if case["kind"] == "post":
        return _exact_post(case, seed)
    return None
