"""The build's radix sort at the edges of its tiles (4096 keys) against the CPU oracle.  Needs a GB300."""
import numpy as np
import pytest
import torch

from gray_gb300 import synthetic
from tests import gpu_util as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spread", ["clustered", "one cell", "two cells"])
@pytest.mark.parametrize("n", [1, 2, 31, 4095, 4096, 4097, 8193, 300_001])
def test_sorted_codes_and_order_match_the_oracle(gray_lib, oracle, n, spread):
    """Codes and order of a build: spread keys, and keys with one or two values (every key of a tile in one
    digit, so the order is the Gaussians' own); a second build on the same scratch gives the same."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sc = synthetic.clustered_scene(n, seed=n % 89)
    mean = sc.mean.copy()
    if spread != "clustered":
        mean[:] = 1.0
        if spread == "two cells":
            mean[::3] = -2.0
    rt = G.make_tracer(8, 8, mean, sc.rotation, sc.scale, sc.opacity, channels=np.full((n, 3), 0.5, np.float32),
                       pool_words=1000)
    _, _, aabb, vis = oracle.snapshot(mean, sc.rotation, sc.scale, sc.opacity.reshape(-1), 0.01)
    tree = oracle.Bvh(aabb, vis)
    ws = rt.scene_workspace()
    for _ in range(2):
        assert np.array_equal(ws.codes.cpu().numpy().view(np.uint32), tree.codes)
        assert np.array_equal(ws.order.cpu().numpy().view(np.uint32), tree.order)
        ws.codes.fill_(-1)
        ws.order.fill_(-1)
        rt.rebuild_bvh()
        rt.check_status()
