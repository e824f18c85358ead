"""Where the cooperative ray cast of a small scene stops taking a chunk's rays from eight places, and where its scene
counts as small: against the grid form, bit for bit (any hit: the same hit or miss)."""
import pytest

import scenes
from test_wide_form_gpu import _check, _rays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level,nodes", [(3, (0, 512)), (4, (512, 1024)), (5, (1024, 1 << 20))])
@pytest.mark.parametrize("extra", [-3, 0, 1, 33])
def test_limit(R, gpu_ctx, level, nodes, extra):
    scene, _, _ = scenes.sphere_scene(R, gpu_ctx, level)
    assert nodes[0] <= scene.stats()["node_count"] < nodes[1]
    n = 700 * gpu_ctx.sm_count + extra
    assert (_check(R, scene, _rays(R, n, n))["prim"] != R.MISS).any()
    scene.close()
