"""The whole-tile kernels against the CPU oracle on dense tiles: variant bit 5 keeps tiles whole that the
schedule would enter as split packets, and the schedule's counts show which kernel had them.  Needs a GB300."""
import numpy as np
import pytest
import torch

from gray_gb300 import synthetic
from tests import gpu_util as G
from tests.test_gpu_parity import _camera_rays_gpu, _compare_forward, _oracle_scene

pytestmark = pytest.mark.gpu

WHOLE, SPLIT, PACKETS, RETRACED, CHOICE = 1, 3, 48, 49, 50  # schedule words
NEVER_SPLIT = 32


@pytest.fixture(scope="module", autouse=True)
def _cuda(gray_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _dense(oracle, size, n, t_threshold, grow):
    W, H = size
    sc = synthetic.small_scene(seed=n, n=n)
    chan = np.random.default_rng(n).uniform(0, 1, (n, 3)).astype(np.float32)
    rt = G.make_tracer(W, H, sc.mean, sc.rotation, sc.scale + np.float32(grow), sc.opacity, channels=chan,
                       t_threshold=t_threshold)
    geom, l2w, aabb, vis, live = _oracle_scene(oracle, sc.mean, sc.rotation, sc.scale + np.float32(grow), sc.opacity)

    def expected(ro, rd):
        return oracle.trace_forward(ro, rd, geom, live, chan, vis, oracle.TraceConfig(t_threshold=t_threshold))
    cam = synthetic.look_at((0.0, -3.0, 0.4), (0, 0, 0), (0, 0, 1), 0.6, W, H)
    return rt, cam, expected


def _tiles(variant, size):
    tile = (8, 16) if variant & 4 else (16, 8)
    return -(-size[0] // tile[0]) * -(-size[1] // tile[1])


@pytest.mark.parametrize("variant", [0, 1, 2, 3, 5, 7])
@pytest.mark.parametrize("size,n,grow", [((8, 16), 127, 0.7), ((9, 17), 128, 0.7), ((16, 9), 129, 0.7),
                                         ((33, 31), 1000, 0.7), ((24, 40), 5000, 0.4)])
@pytest.mark.parametrize("jitter", [False, True])
def test_dense_whole_tiles_match_the_oracle(oracle, variant, size, n, grow, jitter):
    """Tiles of one batch, of one candidate more and of many, over several traversals (rays of more hits than
    16 and 32 slots hold), by the 16- and the 32-slot kernel in both tile shapes."""
    rt, cam, expected = _dense(oracle, size, n, 1e-4, grow)
    rt.get_config().jitter_primary_rays.fill_(jitter)
    rt.set_trace_variant(NEVER_SPLIT + variant)
    ro, rd = _camera_rays_gpu(rt, cam)
    fwd = expected(ro, rd)
    words = rt.schedule[:8].cpu().tolist()
    assert words[WHOLE] == _tiles(variant, size) and words[SPLIT] == 0
    _compare_forward(rt, fwd)
    if n >= 1000:
        assert fwd["nacc"].max() > 32
        # the same tiles are entered as packets otherwise
        rt.set_trace_variant(variant if variant else 4)
        rt.get_stats().reset()
        ro, rd = _camera_rays_gpu(rt, cam)
        words = rt.schedule[:8].cpu().tolist()
        assert words[SPLIT] > 0 and words[WHOLE] + words[SPLIT] // 4 == _tiles(variant if variant else 4, size)
        _compare_forward(rt, expected(ro, rd))


@pytest.mark.parametrize("variant", [3, 7])
def test_supplied_rays_in_whole_tiles_match_the_oracle(oracle, variant):
    """Supplied rays of a cone in whole tiles of many batches."""
    size, n = (40, 36), 3000
    rt, _, expected = _dense(oracle, size, n, 1e-4, 0.4)
    W, H = size
    i, j = np.meshgrid(np.arange(W), np.arange(H))
    x, y = 0.35 * (2 * (i + 0.5) / W - 1), 0.35 * (2 * (j + 0.5) / H - 1)
    d = np.stack([x * (1 + 0.3 * x * x), np.ones_like(x), -y * (1 + 0.3 * y * y)], -1).reshape(-1, 3)
    rd = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    ro = np.tile(np.array([0.1, -3.0, 0.2], np.float32), (W * H, 1))
    fwd = expected(ro, rd)
    assert fwd["nacc"].max() > 32
    for v, split in ((NEVER_SPLIT + variant, False), (variant, True)):
        rt.set_trace_variant(v)
        rt.get_stats().reset()
        G.trace_rays(rt, ro, rd)
        words = rt.schedule[:8].cpu().tolist()
        assert (words[SPLIT] > 0) == split and words[WHOLE] + words[SPLIT] // 4 == _tiles(variant, size)
        _compare_forward(rt, fwd)


@pytest.mark.parametrize("t_threshold", [1e-3, 0.6])
def test_both_whole_tile_kernels_count_the_same_second_traversals(oracle, t_threshold):
    """The packets that need a second traversal with 16 slots, counted by the 16-slot kernel, by the 32-slot
    one and with dense tiles split; the automatic choice follows the small frames' line of 1/128."""
    rt, cam, expected = _dense(oracle, (72, 56), 5000, t_threshold, 0.2)
    counts = {}
    for v in (NEVER_SPLIT + 7, NEVER_SPLIT + 5, 7, 0, 0):
        rt.set_trace_variant(v)
        rt.get_stats().reset()
        ro, rd = _camera_rays_gpu(rt, cam)
        counts[v] = rt.schedule[PACKETS:CHOICE + 1].cpu().tolist()
        split = int(rt.schedule[SPLIT].item())
        assert (split == 0) == (v >= NEVER_SPLIT)
        _compare_forward(rt, expected(ro, rd))
    assert counts[NEVER_SPLIT + 7][0] == counts[NEVER_SPLIT + 5][0] == counts[7][0] == 9 * 4 * 4
    assert counts[NEVER_SPLIT + 7][1] == counts[NEVER_SPLIT + 5][1] == counts[7][1]
    deep = counts[NEVER_SPLIT + 5][1] * 128 > counts[NEVER_SPLIT + 5][0]
    assert deep == (t_threshold < 0.1) and counts[0][2] == (2 if deep else 1)
