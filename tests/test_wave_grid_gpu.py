"""The wave engine's grid form on request, in every block size and stack depth, against the pass-by-pass engine, sample
by sample and bit for bit: with few and with many paths and nodes, flat and two-level scenes, several jobs,
direct launches and graphs.  Without the request these calls run eight lanes per ray or cooperatively."""
import pytest

import scenes
from test_wave_forms_gpu import built, ctx, frame, same, samples   # noqa: F401 (fixtures)

pytestmark = pytest.mark.gpu

VARIANTS = [dict(trace_block=b, trace_stack=s) for b in (64, 128, 256) for s in (8, 12, 16)]


def _grid_forms(R, ctx, jobs):
    try:
        for kw in VARIANTS + [dict(batch_flags=R.BATCH_NO_GRAPHS)]:
            ctx.set_tuning(**{"wave_refill": R.REFILL_GRID_ALWAYS, "batch_flags": 0, "trace_block": 0, "trace_stack": 0, **kw})
            assert ctx.tuning()["wave_refill"] == R.REFILL_GRID_ALWAYS
            yield kw, samples(R, ctx, jobs)
    finally:
        ctx.set_tuning(wave_refill=0, batch_flags=0, trace_block=0, trace_stack=0)


# 301x299 is beyond 352 paths per SM, where flat scenes of many nodes would run cooperatively, and 61x47 below 96
@pytest.mark.parametrize("name", ["few_nodes", "nodes", "textured", "instanced"])
@pytest.mark.parametrize("w,h,spp,mode", [(61, 47, 2, 1), (301, 299, 2, 1), (523, 509, 2, 0)])
def test_variants(R, ctx, built, name, w, h, spp, mode):   # noqa: F811
    s = built[name]
    want = samples(R, ctx, [(s, *frame(R, s, w, h, spp, mode=mode, pass_by_pass=True))])
    for kw, got in _grid_forms(R, ctx, [(s, *frame(R, s, w, h, spp, mode=mode))]):
        same(got, want, kw)


def test_mixed_jobs(R, ctx, built):   # noqa: F811
    jobs, want = [], []
    for name, w, h, spp, bounces, mode in (("nodes", 200, 150, 2, 3, 1), ("instanced", 61, 47, 3, 4, 0), ("glass", 97, 31, 2, 6, 1)):
        jobs.append((built[name], *frame(R, built[name], w, h, spp, bounces, mode)))
        want += samples(R, ctx, [(built[name], *frame(R, built[name], w, h, spp, bounces, mode, pass_by_pass=True))])
    for kw, got in _grid_forms(R, ctx, jobs):
        same(got, want, kw)


@pytest.mark.parametrize("name", ["few_nodes", "nodes"])
def test_chosen_grid_variants(R, ctx, built, name):   # noqa: F811
    """Block sizes and stack depths where the engine itself chooses the form (few nodes: the grid form)."""
    s = built[name]
    want = samples(R, ctx, [(s, *frame(R, s, 301, 299, 2, pass_by_pass=True))])
    try:
        for kw in VARIANTS:
            ctx.set_tuning(wave_refill=0, **kw)
            same(samples(R, ctx, [(s, *frame(R, s, 301, 299, 2))]), want, kw)
    finally:
        ctx.set_tuning(trace_block=0, trace_stack=0)
