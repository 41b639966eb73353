"""The backward's sums per hit and the pass that carries them to the parameters, against the CPU oracle.
Needs a GB300."""
import numpy as np
import pytest
import torch

from gray_gb300 import synthetic
from tests import gpu_util as G
from tests.test_gpu_parity import GRAD_RTOL, _camera_rays_gpu, _grad_close, _oracle_scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda(gray_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("exp_power", [1.0, 2.0, 3.0])
@pytest.mark.parametrize("n", [1, 127, 512, 513, 1500])
def test_gradients_of_stretched_gaussians_match_the_oracle(oracle, n, exp_power):
    """Axis ratios of up to 1:90, counts around the rows a block of the fold lists, two backward passes on top
    of one another.  The bar is the one of the reference scenes: the oracle accumulates in 64 bits, and 32-bit
    sums of at most a few thousand hits stay within 1e-4 of the largest gradient."""
    W, H = 33, 21
    rng = np.random.default_rng(n)
    sc = synthetic.small_scene(seed=n, n=n)
    scale = rng.uniform(-5.0, -0.5, (n, 3)).astype(np.float32) + np.float32(1.0 if n == 1 else 0.0)
    mean = (sc.mean * np.float32(0.0 if n == 1 else 1.0)).astype(np.float32)
    opacity = rng.uniform(-2.0, 4.0, n).astype(np.float32)
    chan = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    rt = G.make_tracer(W, H, mean, sc.rotation, scale, opacity, channels=chan, exp_power=exp_power,
                       bg=(0.2, 0.5, 0.1))
    cam = synthetic.look_at((0.0, -3.0, 0.4), (0, 0, 0), (0, 0, 1), 0.6, W, H)
    ro, rd = _camera_rays_gpu(rt, cam)
    rt.check_status()
    geom, l2w, aabb, vis, live = _oracle_scene(oracle, mean, sc.rotation, scale, opacity, p=exp_power)
    cfg = oracle.TraceConfig(exp_power=exp_power, bg=(0.2, 0.5, 0.1))
    fwd = oracle.trace_forward(ro, rd, geom, live, chan, vis, cfg)
    gout = rng.normal(0, 1, (H * W, 3)).astype(np.float32)
    ref = oracle.trace_backward(W, H, ro, rd, fwd, gout, geom, l2w, opacity, scale, sc.rotation, chan, cfg)
    assert ref[:, 15].sum() > 0
    g = rt.get_gaussians()
    for times in (1, 2):
        rt.get_framebuffer().grad_output_channels.copy_(torch.from_numpy(gout).reshape(H, W, 3))
        rt.backward_pass()
        torch.cuda.synchronize()
        rt.check_status()
        for t, sl in ((g.grad_rotation, slice(0, 4)), (g.grad_mean, slice(4, 7)), (g.grad_opacity, slice(7, 8)),
                      (g.grad_scale, slice(8, 11)), (g.grad_channels, slice(12, 15))):
            _grad_close(t.cpu().numpy(), times * ref[:, sl], GRAD_RTOL)
        _grad_close(g.pruning_weight.cpu().numpy(), times * ref[:, 11:12], GRAD_RTOL)
        assert np.array_equal(g.was_visible.cpu().numpy()[:, 0], ref[:, 15] > 0)
    assert not rt.scene_workspace().grad_acc.any()
