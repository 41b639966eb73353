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


def _supplied_rays(kind, W, H, rng):
    """Rays of a lens the pinhole camera does not have: [W*H, 3] origins and directions."""
    i, j = np.meshgrid(np.arange(W), np.arange(H))
    o = np.tile(np.array([0.1, -3.5, 0.2], np.float32), (W * H, 1))
    if kind == "panorama":  # the whole sphere: tiles near the poles are too wide for a cone
        az, el = 2 * np.pi * (i + 0.5) / W, np.pi * ((j + 0.5) / H - 0.5)
        d = np.stack([np.cos(el) * np.sin(az), np.cos(el) * np.cos(az), np.sin(el)], -1)
    else:
        x, y = 0.9 * (2 * (i + 0.5) / W - 1), 0.9 * (2 * (j + 0.5) / H - 1)
        bend = 1.0 + 0.3 * (x * x + y * y)
        d = np.stack([x * bend * 0.3, np.ones_like(x), -y * bend * 0.3], -1)
    d = (d / np.linalg.norm(d, axis=-1, keepdims=True)).reshape(-1, 3)
    if kind == "lengths":
        d *= 2.0 ** rng.uniform(-3, 3, (W * H, 1))
    elif kind == "extreme lengths":
        d *= 2.0 ** rng.choice([-14.0, 0.0, 14.0], (W * H, 1))
    elif kind == "holes":
        d[rng.random(W * H) < 0.4] = 0.0
        d[: 8 * W] = 0.0
    elif kind == "origins":  # one row of tiles with an origin per ray, the others with one each
        o = o + np.repeat(0.02 * (np.arange(H) // 16).astype(np.float32), W)[:, None]
        o[: 16 * W] += 0.05 * rng.standard_normal((16 * W, 3))
    elif kind == "parallel":
        d[:] = np.array([0.02, 1.0, -0.03]) / np.linalg.norm([0.02, 1.0, -0.03])
    elif kind == "shuffled":  # neighbouring pixels' rays all over the image
        d = d[rng.permutation(W * H)]
    return o.astype(np.float32), d.astype(np.float32)


@pytest.mark.parametrize("kind", ["lens", "panorama", "lengths", "extreme lengths", "holes", "origins", "parallel",
                                  "shuffled"])
def test_rays_from_the_caller_match_the_oracle(oracle, kind):
    """Supplied rays are traversed tile by tile where a tile's rays share their origin and a cone, and one
    by one elsewhere: images, hit lists and counts are the oracle's either way."""
    W, H, n = 45, 39, 1500
    rng = np.random.default_rng(5)
    sc = synthetic.small_scene(seed=n, n=n)
    grow = np.float32(0.4)
    chan = np.random.default_rng(n).uniform(0, 1, (n, 3)).astype(np.float32)
    rt = G.make_tracer(W, H, sc.mean, sc.rotation, sc.scale + grow, sc.opacity, channels=chan)
    geom, l2w, aabb, vis, live = _oracle_scene(oracle, sc.mean, sc.rotation, sc.scale + grow, sc.opacity)
    ro, rd = _supplied_rays(kind, W, H, rng)
    for _ in range(2):
        rt.get_stats().reset()
        G.trace_rays(rt, ro, rd)
        fwd = oracle.trace_forward(ro, rd, geom, live, chan, vis, oracle.TraceConfig(t_threshold=0.03))
        assert fwd["nhit"].max() > 3
        _compare_forward(rt, fwd)


@pytest.mark.parametrize("size", [(9, 17), (64, 48), (130, 70)])
def test_jittered_tiles_match_the_oracle(oracle, size):
    """Jittered camera rays are traversed tile by tile, up to half a pixel beyond the pixels' centres."""
    W, H = size
    n = 3000
    sc = synthetic.small_scene(seed=n, n=n)
    chan = np.random.default_rng(n).uniform(0, 1, (n, 3)).astype(np.float32)
    rt = G.make_tracer(W, H, sc.mean, sc.rotation, sc.scale, sc.opacity, channels=chan, t_threshold=1e-3)
    rt.get_config().jitter_primary_rays.fill_(True)
    cam = synthetic.look_at((0.0, -3.0, 0.4), (0, 0, 0), (0, 0, 1), 0.6, W, H)
    geom, l2w, aabb, vis, live = _oracle_scene(oracle, sc.mean, sc.rotation, sc.scale, sc.opacity)
    for _ in range(2):
        rt.get_stats().reset()
        ro, rd = _camera_rays_gpu(rt, cam)
        fwd = oracle.trace_forward(ro, rd, geom, live, chan, vis, oracle.TraceConfig(t_threshold=1e-3))
        _compare_forward(rt, fwd)


@pytest.mark.parametrize("offsets", ["numbered", "gap", "none"])
def test_ordered_batch_equals_plain_views(offsets):
    """A batch with more than four groups per block renders its densest groups first; views whose group
    offsets do not number the groups one after another, or no frontier at all, keep the views' order.  The
    pixels are the plain forward's in every case."""
    import ctypes

    from gray_gb300.batch import BatchRenderer, BatchViewC

    sc = synthetic.clustered_scene(20_000, seed=3)
    rt = G.make_tracer(640, 480, sc.mean, sc.rotation, sc.scale, sc.opacity,
                       channels=np.random.default_rng(1).uniform(0, 1, (sc.n, 3)).astype(np.float32))
    cams = [synthetic.orbit_camera(0.9 * k, w, h) for k, (w, h) in enumerate(((640, 480), (633, 471), (640, 480)))]
    br = BatchRenderer([rt], use_graph=False, autotune=False, variant=5, blocks_per_sm=1)
    reqs = [(0, c) for c in cams]
    br.render(reqs)
    plan = next(iter(br.plans.values()))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert plan.total_groups > 4 * sms
    if offsets == "gap":
        views = (BatchViewC * 3).from_buffer(plan.views_host.numpy())
        views[2].group_offset += 1
    if offsets == "none":
        plan.total_groups = 0
    plan.out.zero_()
    br._launch(plan)
    br.check_status()
    for i, c in enumerate(cams):
        rt.set_render_resolution(c.image_width, c.image_height)
        rt.set_view(c.origin_cuda(), c.rotation_c2w_blender_cuda(), c.fov_y, 0.0, 99999.9)
        rt.forward_pass_display()
        plain = rt.get_framebuffer().output_channels[:c.image_height, :c.image_width]
        got = plan.out[plan.offsets[i]:plan.offsets[i] + plain.numel()].view(plain.shape)
        assert torch.equal(got, plain), i
