"""Autotuning a frame beside the wave engine's own choice of form: another configuration is taken only where it is faster
by more than timings differ, and a cached entry leaves images as they are, for calls it holds for and others."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def _call(R, scene, side, spp, mode):
    iv, ip = scenes.cornell_camera(R, side, side)
    pc = R.push_consts(iv, ip, total_emissive_weight=scene.emissive_weight, spp=spp, max_bounces=5, focus_dist=3.4)
    return pc, R.render_options(side, side, mode, 3)


@pytest.mark.parametrize("level", [1, 5])
@pytest.mark.parametrize("side,spp,mode", [(48, 1, 1), (48, 3, 0), (300, 2, 1)])
def test_default_kept_within_noise(R, level, side, spp, mode):
    """Few paths run eight lanes per ray and scenes of 512 or more nodes cooperatively, whatever the grid form's block size
    and stack depth: a tuner that timed those all the same would keep the winner of noise."""
    ctx = R.Context(0)
    d = scenes.cornell(R)
    v, i, tbn, ti = scenes.sphere_tbn(level, 0.1, 3, R)
    d.add_instance(d.add_object(v, i, tbn, ti), scenes.scale(0.6, 0.6, 0.6), R.Material())
    s = d.to_product(R, ctx)
    pc, opts = _call(R, s, side, spp, mode)
    want, _, _ = R.render(ctx, s, pc, opts)
    default = {k: ctx.tuning()[k] for k in ("wave_refill", "trace_block", "trace_stack")}
    for _ in range(4):
        res = R.autotune_render(ctx, s, pc, opts)
        assert res["candidates"] == 12
        best = {k: res["best"][k] for k in default}
        assert best == default or res["best_ms"] <= 0.98 * res["default_ms"], res
        assert res["best"]["wave_paths"] == ctx.tuning()["wave_paths"]
    R.autotune_set_mode(ctx, R.AUTOTUNE_CACHED)
    assert np.array_equal(R.render(ctx, s, pc, opts)[0], want)
    s.close()
    ctx.close()


@pytest.mark.parametrize("refill", [-1, 0, 8])
@pytest.mark.parametrize("paths", [0, 1, 2304, 1 << 20])
def test_cached_entries(R, tmp_path, refill, paths):
    """Entries for any call, for pass-by-pass frames, for calls like this one and for larger ones."""
    ctx = R.Context(0)
    s = scenes.material_zoo(R).to_product(R, ctx)
    p = tmp_path / "t.txt"
    tris = s.stats()["triangle_count"]
    p.write_text(f"2 {tris.bit_length() - 1} {(48 * 48).bit_length() - 1} {refill} 64 16 {paths} 1 1\n")
    for mode, spp in ((0, 1), (1, 1), (1, 500)):
        pc, opts = _call(R, s, 48, spp, mode)
        R.autotune_set_mode(ctx, R.AUTOTUNE_OFF)
        want, _, _ = R.render(ctx, s, pc, opts)
        R.autotune_load(ctx, p)
        R.autotune_set_mode(ctx, R.AUTOTUNE_CACHED)
        for kw in (dict(), dict(pass_by_pass=True)):
            got, _, _ = R.render(ctx, s, pc, R.render_options(48, 48, mode, 3, **kw))
            assert np.array_equal(got, want, equal_nan=True), (mode, spp, kw, np.argwhere(got != want)[:5])
    s.close()
    ctx.close()
