"""The device BVH builder at the task sizes where it changes path: 8 lanes or a warp per task (8 primitives),
a warp or work items (512), one or several work items (256), and 32 or more SAH bins (one or two rounds of
the sweeps).  Same bytes as the host builder."""
import numpy as np
import pytest

from test_bvh_device_gpu import _same, _soup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [6, 7, 8, 10, 17, 64, 257, 511, 512, 513, 769, 1025, 5000])
@pytest.mark.parametrize("bins,median_depth", [(0, 0), (33, 0), (64, 5), (4, 2), (0, 1)])
def test_task_sizes(R, gpu_ctx, n, bins, median_depth):
    v, i = _soup(n, seed=n + bins)
    _same(R, gpu_ctx, v, i, bins, median_depth)


@pytest.mark.parametrize("n", [5, 8, 9, 40, 600])
def test_repeated_and_axis_aligned(R, gpu_ctx, n):
    """Clusters of equal triangles (medians inside tiny tasks) on a line with signed zeros (two axes cannot be
    binned)."""
    g = np.random.default_rng(n)
    v = np.zeros((3 * n, 3), np.float32)
    x = np.repeat(g.integers(0, max(2, n // 4), n).astype(np.float32), 3)
    v[:, 0] = x + np.tile(np.float32([0.0, 0.5, 0.0]), n)
    v[1::3, 1] = 1.0
    v[::2, 2] = -0.0
    _same(R, gpu_ctx, v, np.arange(3 * n, dtype=np.uint32))
