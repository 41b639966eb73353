"""The cone of a tile of the caller's rays, built by the block that traces it, against the CPU oracle where the
block's warps differ: some without rays, one with a ray that spoils the cone.  Needs a GB300."""
import numpy as np
import pytest
import torch

from gray_gb300 import synthetic
from tests import gpu_util as G
from tests.test_gpu_parity import _compare_forward, _oracle_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["all", "last warp", "second warp", "one ray", "origin in the last warp",
                                  "length in the third warp", "wide in the first warp"])
@pytest.mark.parametrize("size", [(8, 16), (20, 45)])
def test_cones_of_uneven_tiles(oracle, gray_lib, kind, size):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    (W, H), n = size, 5000
    sc = synthetic.small_scene(seed=n, n=n)
    grow = np.float32(0.0)
    chan = np.random.default_rng(n).uniform(0, 1, (n, 3)).astype(np.float32)
    rt = G.make_tracer(W, H, sc.mean, sc.rotation, sc.scale + grow, sc.opacity, channels=chan, t_threshold=1e-3)
    geom, l2w, aabb, vis, live = _oracle_scene(oracle, sc.mean, sc.rotation, sc.scale + grow, sc.opacity)
    i, j = np.meshgrid(np.arange(W), np.arange(H))
    d = np.stack([0.3 * (2 * (i + 0.5) / W - 1), np.ones((H, W)), -0.3 * (2 * (j + 0.5) / H - 1)], -1)
    d /= np.linalg.norm(d, axis=-1, keepdims=True)
    o = np.broadcast_to(np.array([0.1, -3.0, 0.2]), d.shape).copy()
    part = (j % 16) * 8 + i % 8  # a whole tile's ray by its thread
    if kind == "last warp":
        d[part < 96] = 0.0
    elif kind == "second warp":
        d[(part < 32) | (part >= 64)] = 0.0
    elif kind == "one ray":
        d[part != 77] = 0.0
    elif kind == "origin in the last warp":
        o[part == 120] += 0.125
    elif kind == "length in the third warp":
        d[part == 70] *= 4096.0
    elif kind == "wide in the first warp":
        d[part == 5] *= -1.0
    ro, rd = o.reshape(-1, 3).astype(np.float32), d.reshape(-1, 3).astype(np.float32)
    fwd = oracle.trace_forward(ro, rd, geom, live, chan, vis, oracle.TraceConfig(t_threshold=1e-3))
    assert fwd["nhit"].max() > 8
    for _ in range(2):
        rt.get_stats().reset()
        G.trace_rays(rt, ro, rd)
        _compare_forward(rt, fwd)
    # no super-tile walks: the caller's rays are read by their tiles alone
    tiles = -(-W // 8) * -(-H // 16)
    frontier = int(gray_lib.gray_frontier_words())
    supers = rt.schedule[64 + tiles * (6 + frontier):][:1].cpu().numpy().view(np.uint32)
    assert supers[0] == 0xFFFFFFFF
