"""Which of the caller's rays are traversed tile by tile and which one by one, and that both give the CPU
oracle's results.  Needs a GB300."""
import numpy as np
import pytest
import torch

from gray_gb300 import synthetic
from tests import gpu_util as G
from tests.test_gpu_parity import _compare_forward, _oracle_scene

pytestmark = pytest.mark.gpu

WHOLE, SPLIT, SINGLE = 1, 3, 4  # schedule words: whole tiles, packets of split tiles, tiles of single rays


@pytest.fixture(scope="module", autouse=True)
def _cuda(gray_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _rays(kind, W, H, distance, rng):
    i, j = np.meshgrid(np.arange(W), np.arange(H))
    o = np.tile(np.array([0.1, -distance, 0.2], np.float32), (W * H, 1))
    if kind == "mosaic":  # thumbnails of 16x16 rays, each of the whole view
        x, y = 0.5 * (2 * (i % 16 + 0.5) / 16 - 1), 0.5 * (2 * (j % 16 + 0.5) / 16 - 1)
    else:
        x, y = 0.5 * W / H * (2 * (i + 0.5) / W - 1), 0.5 * (2 * (j + 0.5) / H - 1)
    d = np.stack([x, np.ones_like(x), -y], -1).reshape(-1, 3)
    d /= np.linalg.norm(d, axis=-1, keepdims=True)
    if kind == "shuffled":  # every tile's rays all over the view
        d = d[rng.permutation(W * H)]
    elif kind == "origins":
        o = o + 0.05 * rng.standard_normal((W * H, 3)).astype(np.float32)
    elif kind == "half origins":  # tiles of both kinds in one frame
        o[(np.arange(W * H) // W) < 16 * (H // 32)] += np.float32(0.25)
        own = (np.arange(W * H) // W) >= 16 * (H // 32)
        o[own] += 0.05 * rng.standard_normal((int(own.sum()), 3)).astype(np.float32)
    return o.astype(np.float32), d.astype(np.float32)


def _scene(kind, n):
    if kind == "clustered":
        return synthetic.clustered_scene(n, seed=5), 8.0
    return synthetic.small_scene(seed=n, n=n), 3.5


# the tiles of each frame that are traversed one by one: none, all, or those with an origin per ray
@pytest.mark.parametrize("scene,n,size,kind,single", [
    ("small", 128, (33, 20), "pinhole", "all"),
    ("small", 129, (33, 20), "pinhole", "none"),
    ("small", 1500, (45, 39), "pinhole", "none"),
    ("small", 1500, (45, 39), "origins", "all"),
    ("small", 1500, (45, 64), "half origins", "half"),
    ("small", 1500, (45, 39), "shuffled", "none"),
    ("clustered", 60_000, (64, 48), "pinhole", "none"),
    ("clustered", 60_000, (64, 48), "origins", "all"),
    ("clustered", 60_000, (64, 48), "shuffled", "all"),
    ("clustered", 60_000, (192, 256), "mosaic", "all"),
])
def test_routes_of_supplied_rays(oracle, scene, n, size, kind, single):
    """Tiny scenes, origins of their own and tiles that few of their rays' candidates are met in (rays of a
    clustered scene shuffled over the view, or thumbnails) go one by one."""
    W, H = size
    sc, distance = _scene(scene, n)
    chan = np.random.default_rng(n).uniform(0, 1, (n, 3)).astype(np.float32)
    rt = G.make_tracer(W, H, sc.mean, sc.rotation, sc.scale, sc.opacity, channels=chan, t_threshold=1e-3)
    geom, l2w, aabb, vis, live = _oracle_scene(oracle, sc.mean, sc.rotation, sc.scale, sc.opacity)
    ro, rd = _rays(kind, W, H, distance, np.random.default_rng(3))
    fwd = oracle.trace_forward(ro, rd, geom, live, chan, vis, oracle.TraceConfig(t_threshold=1e-3),
                               bvh=oracle.Bvh(aabb, vis) if scene == "clustered" else None)
    tx, ty = -(-W // 8), -(-H // 16)
    for _ in range(2):
        rt.get_stats().reset()
        G.trace_rays(rt, ro, rd)
        words = rt.schedule[:8].cpu().tolist()
        assert words[WHOLE] + words[SPLIT] // 4 + words[SINGLE] == tx * ty
        assert words[SINGLE] == {"none": 0, "all": tx * ty, "half": tx * (ty - H // 32)}[single], words
        _compare_forward(rt, fwd)


@pytest.mark.parametrize("n", [400, 20_000])
def test_rays_composite_more_hits_than_a_buffer_holds(oracle, n):
    """Single rays of more hits than their 32 slots hold: several traversals, several list segments."""
    W, H = 24, 40
    sc = synthetic.small_scene(seed=n, n=n)
    grow = np.float32(2.0 if n < 1000 else 0.0)
    chan = np.random.default_rng(n).uniform(0, 1, (n, 3)).astype(np.float32)
    opacity = sc.opacity - np.float32(2.0)
    rt = G.make_tracer(W, H, sc.mean, sc.rotation, sc.scale + grow, opacity, channels=chan, t_threshold=1e-4)
    geom, l2w, aabb, vis, live = _oracle_scene(oracle, sc.mean, sc.rotation, sc.scale + grow, opacity)
    ro, rd = _rays("origins", W, H, 3.5, np.random.default_rng(4))
    fwd = oracle.trace_forward(ro, rd, geom, live, chan, vis, oracle.TraceConfig(t_threshold=1e-4))
    assert fwd["nacc"].max() > 64
    G.trace_rays(rt, ro, rd)
    assert rt.schedule[SINGLE].item() == 9
    _compare_forward(rt, fwd)
