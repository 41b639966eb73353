"""Which tiles a forward enters as split packets: the schedule's counts against the rule computed from its own
estimates.  Needs a GB300."""
import numpy as np
import pytest
import torch

from gray_gb300 import synthetic
from tests import gpu_util as G

pytestmark = pytest.mark.gpu

HEADER, WHOLE, SPLIT, CHOICE = 64, 1, 3, 50


def expected_split(est, slots):
    """The number of tiles that are split."""
    est = np.asarray(est, np.int64)
    above = max(96, int(est.sum()) * 5 // (8 * slots))
    dense = np.sort(est[est > above])[::-1]
    limit = slots // 12 if est.size <= slots else slots // 6
    steep = 5 if int(est.max()) >= 16384 else 10
    if est.size <= slots // 4 or 2 * int(est.max()) * slots >= steep * int(est.sum()):
        limit = dense.size
    if dense.size <= limit:
        return dense.size
    octave = np.floor(np.log2(dense)).astype(np.int64)
    edge = (dense >> (octave - 2)) << (octave - 2)  # the lower edge of each one's quarter octave
    return max((int((dense >= e).sum()) for e in edge if (dense >= e).sum() <= limit), default=0)


@pytest.mark.parametrize("scene,n,size,distance", [
    ("small", 1000, (160, 120), 2.2), ("small", 10_000, (160, 120), 4.0), ("small", 10_000, (320, 240), 2.2),
    ("small", 10_000, (320, 240), 4.0), ("small", 10_000, (640, 480), 4.0), ("small", 3000, (480, 360), 2.2),
    ("clustered", 200_000, (160, 120), 8.0), ("clustered", 200_000, (320, 240), 8.0),
    ("clustered", 200_000, (640, 480), 8.0), ("clustered", 500_000, (480, 360), 8.0),
    ("clustered", 500_000, (1280, 720), 8.0), ("clustered", 1_000_000, (320, 240), 12.0),
    ("clustered", 3_000_000, (480, 360), 8.0)])
def test_split_tiles_follow_the_rule(gray_lib, scene, n, size, distance):
    """Few tiles, as many as resident blocks, more; tiles alike (none split), a few dense ones, one far denser
    than the average."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    W, H = size
    sc = synthetic.clustered_scene(n, seed=3) if scene == "clustered" else synthetic.small_scene(seed=n, n=n)
    rt = G.make_tracer(W, H, sc.mean, sc.rotation, sc.scale, sc.opacity, inference_only=True,
                       channels=np.zeros((sc.n, 3), np.float32))
    cam = synthetic.look_at((0.6 * distance, -0.8 * distance, 0.2), (0, 0, 0), (0, 0, 1), 0.9, W, H)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles = -(-W // 8) * -(-H // 16)
    for variant, slots in ((0, None), (7, 5 * sms), (5, 4 * sms), (32 + 7, 0)):
        rt.set_trace_variant(variant)
        rt.set_view(cam.origin_cuda(), cam.rotation_c2w_blender_cuda(), cam.fov_y, 0.0, 99999.9)
        for _ in range(2):
            rt.forward_pass_display()
        words = rt.schedule[:HEADER + tiles].cpu().tolist()
        if slots is None:
            slots = (4 if words[CHOICE] == 2 else 5) * sms
        want = expected_split(words[HEADER:], slots) if slots else 0
        assert words[SPLIT] == 4 * want and words[WHOLE] == tiles - want, (variant, want, words[SPLIT] // 4)


@pytest.mark.parametrize("size", [(160, 120), (320, 240)])
def test_split_tiles_of_supplied_rays(gray_lib, size):
    """Thumbnails, every tile alike: all split in a frame of up to two tiles per SM, none in a larger one."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    W, H = size
    n = 10_000
    sc = synthetic.small_scene(seed=n, n=n)
    rt = G.make_tracer(W, H, sc.mean, sc.rotation, sc.scale, sc.opacity, inference_only=True,
                       channels=np.zeros((n, 3), np.float32))
    i, j = np.meshgrid(np.arange(W), np.arange(H))
    x, y = 0.2 * (2 * (i % 16 + 0.5) / 16 - 1), 0.2 * (2 * (j % 16 + 0.5) / 16 - 1)
    d = np.stack([x, np.ones_like(x), -y], -1).reshape(-1, 3)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    G.trace_rays(rt, np.tile(np.array([0.1, -3.5, 0.2]), (W * H, 1)), d, grads=False)
    tiles = -(-W // 8) * -(-H // 16)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    words = rt.schedule[:HEADER + tiles].cpu().tolist()
    assert words[4] == 0  # none one by one
    assert words[SPLIT] == (4 * tiles if tiles <= 2 * sms else 0), (words[:6], min(words[HEADER:]), max(words[HEADER:]))
