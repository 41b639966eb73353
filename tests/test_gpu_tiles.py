"""The forward's block tiles against the CPU oracle, bit for bit, at the sizes where a tile, a batch of
candidates or the traversal's stack and queue can go wrong.  Needs a GB300."""
import numpy as np
import pytest
import torch

from gray_gb300 import synthetic
from tests import gpu_util as G
from tests.test_gpu_parity import _camera_rays_gpu, _compare_forward, _oracle_scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda(gray_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("variant", [0, 1, 2, 3, 7, 31])
@pytest.mark.parametrize("size,n", [((1, 1), 1), ((8, 16), 2), ((9, 17), 127), ((7, 33), 128), ((40, 15), 129),
                                    ((16, 8), 300), ((33, 31), 1000), ((24, 40), 5000)])
def test_tiles_match_the_oracle(oracle, variant, size, n):
    """Scenes whose tiles reach fewer, exactly and more candidates than a batch holds, on images smaller
    than a tile, exact multiples of it and one pixel beyond; the last ones composite over several
    traversals."""
    W, H = size
    sc = synthetic.small_scene(seed=n, n=n)
    grow = np.float32(0.0 if n < 1000 else 0.7)
    chan = np.random.default_rng(n).uniform(0, 1, (n, 3)).astype(np.float32)
    rt = G.make_tracer(W, H, sc.mean, sc.rotation, sc.scale + grow, sc.opacity, channels=chan, t_threshold=1e-4)
    rt.set_trace_variant(variant)
    cam = synthetic.look_at((0.0, -3.0, 0.4), (0, 0, 0), (0, 0, 1), 0.6, W, H)
    geom, l2w, aabb, vis, live = _oracle_scene(oracle, sc.mean, sc.rotation, sc.scale + grow, sc.opacity)
    for _ in range(2):  # the second forward follows the first one's statistics
        rt.get_stats().reset()
        ro, rd = _camera_rays_gpu(rt, cam)
        rt.check_status()
        fwd = oracle.trace_forward(ro, rd, geom, live, chan, vis, oracle.TraceConfig(t_threshold=1e-4))
        _compare_forward(rt, fwd)
