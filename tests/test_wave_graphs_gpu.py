"""The wave engine keeps the captured graphs of its waves within a bound: a program whose frames change shape goes on
without its memory growing, and a shape that has been given up renders the same when it comes back."""
import numpy as np
import pytest
import torch

import scenes

pytestmark = pytest.mark.gpu


def _frame(R, ctx, scene, bounces, d):
    iv, ip = scenes.cornell_camera(R, 16, 16)
    pc = R.push_consts(iv, ip, total_emissive_weight=scene.emissive_weight, spp=1, max_bounces=bounces, focus_dist=3.4)
    R.render_device(ctx, scene, pc, R.render_options(16, 16, R.MODE_NEE_MIS, 7), d.data_ptr())
    torch.cuda.synchronize()
    return d.cpu().numpy().copy()


def test_memory_of_changing_shapes(R):
    ctx = R.Context(0)
    scene = scenes.cornell(R).to_product(R, ctx)
    d = torch.zeros((16, 16, 4), device="cuda")
    first = _frame(R, ctx, scene, 60, d)
    for b in range(61, 80):   # 1,330 bounces in all: more than are kept
        _frame(R, ctx, scene, b, d)
    before = torch.cuda.mem_get_info()[0]
    for b in range(80, 130):   # another 5,225 bounces: 680 MB if all were kept
        _frame(R, ctx, scene, b, d)
    assert before - torch.cuda.mem_get_info()[0] < 64 << 20
    assert np.array_equal(_frame(R, ctx, scene, 60, d), first)
    assert np.array_equal(_frame(R, ctx, scene, 1500, d), _frame(R, ctx, scene, 1500, d))   # alone above the bound
    assert np.array_equal(_frame(R, ctx, scene, 60, d), first)
    scene.close()
    ctx.close()
