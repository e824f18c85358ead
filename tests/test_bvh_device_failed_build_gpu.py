"""A device build that fails gives the memory of what it had uploaded back at once, while the scene is still there."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("two_level", [False, True])
def test_memory_of_a_failed_build(R, gpu_ctx, two_level):
    n = 300_000
    g = np.random.default_rng(1)
    v = np.ones((3 * n, 4), np.float32)
    v[:, :3] = (g.uniform(-1, 1, (n, 1, 3)) + 0.01 * g.standard_normal((n, 3, 3))).reshape(-1, 3)
    v[-1, 0] = np.inf
    s = R.Scene(gpu_ctx)
    s.set_bvh_build(R.BVH_DEVICE, 0)
    s.set_accel(R.ACCEL_TWO_LEVEL if two_level else R.ACCEL_FLAT)
    s.add_object(v, np.arange(3 * n, dtype=np.uint32))
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(2):   # its tables take 30 MB
        with pytest.raises(R.ReinaError, match="non-finite|invalid box"):
            s.build()
        assert before - torch.cuda.mem_get_info()[0] < 8 << 20
    s.close()
