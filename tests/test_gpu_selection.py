"""The selection buffer against the CPU oracle where a hit's distance is negative zero.  Needs a GB300."""
import numpy as np
import pytest
import torch

from gray_gb300 import synthetic
from tests import gpu_util as G
from tests.test_gpu_parity import _compare_forward, _oracle_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 1, 7])
@pytest.mark.parametrize("znear", [0.0, -1.0])
def test_rays_that_start_at_a_gaussians_centre(oracle, gray_lib, variant, znear):
    """The Gaussian at the rays' origin is hit at the distance -0, whose key sorts after every other one's.
    With a negative znear it is kept, and the hits beyond a full buffer that holds it are still nearer."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    W, H, n = 24, 20, 400
    sc = synthetic.small_scene(seed=n, n=n)
    mean = sc.mean.copy()
    mean[7] = (0.125, -2.5, 0.25)
    scale = sc.scale + np.float32(1.2)
    chan = np.random.default_rng(n).uniform(0, 1, (n, 3)).astype(np.float32)
    rt = G.make_tracer(W, H, mean, sc.rotation, scale, sc.opacity, channels=chan, t_threshold=1e-4)
    rt.set_trace_variant(variant)
    rt.get_camera().znear.fill_(znear)
    geom, l2w, aabb, vis, live = _oracle_scene(oracle, mean, sc.rotation, scale, sc.opacity)
    i, j = np.meshgrid(np.arange(W), np.arange(H))
    d = np.stack([0.5 * (2 * (i + 0.5) / W - 1), np.ones((H, W)), -0.4 * (2 * (j + 0.5) / H - 1)], -1).reshape(-1, 3)
    rd = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    ro = np.tile(mean[7], (W * H, 1)).astype(np.float32)
    cfg = oracle.TraceConfig(t_threshold=1e-4, znear=znear)
    fwd = oracle.trace_forward(ro, rd, geom, live, chan, vis, cfg)
    assert fwd["nacc"].max() > 32 and bool((fwd["ids"] == 7).any()) == (znear < 0.0)
    for _ in range(2):
        rt.get_stats().reset()
        G.trace_rays(rt, ro, rd)
        _compare_forward(rt, fwd)
