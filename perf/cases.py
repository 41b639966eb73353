"""Performance cases: the calls that a user of gray_gb300 makes, over the range of sizes they are made at.

A case names one kind of call and its sizes:

  render   Raytracer.__call__ without gradients: a view of a trained scene (camera upload, colours,
           trace, image).  half: fp16 SH coefficients, as an inference-only tracer stores them.
  display  the serving loop's request: a resident fp32 scene, camera upload, forward_pass_display.
  rays     forward_pass on rays that the caller supplies (rays_from_python), with depth.
  batch    BatchRenderer.render: many uneven views of one scene in one launch.
  train    one training iteration: render with gradients, L1 loss, backward, step (Adam + refit).
  grad     gray_gb300.autograd.render and its backward: gradients for an optimiser of the caller's own.
  optim    Raytracer.step alone: pruning statistics, Adam over every parameter, snapshot and refit.
  rebuild  rebuild_bvh: after loading, pruning or densifying a scene.

Scenes are seeded stand-ins with the distributions of gray_gb300.synthetic: "box" (a few Gaussians in
a unit box) below 20 000 Gaussians and "clustered" (200 anisotropic clusters in a radius-10 ball) above.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import gray_gb300 as gray
from gray_gb300 import autograd as gray_autograd
from gray_gb300 import classes, synthetic
from gray_gb300.batch import BatchRenderer
from gray_gb300.camera import CameraInfo, look_at

BOX_BELOW = 20_000
MAX_ALPHA = 0.9999
ALPHA_MIN = 0.01          # RaytracerConfig.alpha_threshold
T_MIN = 0.03              # RaytracerConfig.t_threshold
# learning rates of the end of a training run (the decayed ones), so that a scene stays what it is over
# many passes
LATE_RATES = dict(mean=1.6e-6, rotation=1e-5, scale=5e-5, opacity=2.5e-4, sh_dc=2.5e-5, sh_rest=1.25e-6)
PARAMS = ("mean", "rotation", "scale", "opacity", "sh_coeffs_dc", "sh_coeffs_rest")


def listed():
    return [
        # the smallest scene of the test-suite: launches and latency are all there is
        dict(name="render-64-256x256", kind="render", n=64, width=256, height=256, degree=3, half=False, orbit="plain"),
        # a preview of a medium scene with fp16 coefficients, the inference form
        dict(name="render-500k-640x480-half", kind="render", n=500_000, width=640, height=480, degree=3, half=True,
             orbit="plain"),
        # render-only forward at the benchmark's size
        dict(name="render-3m-1080p", kind="render", n=3_000_000, width=1920, height=1080, degree=3, half=False,
             orbit="plain"),
        # the largest request of the serving workload, on a jittered orbit pose
        dict(name="display-6m-4k", kind="display", n=6_000_000, width=3840, height=2160, degree=3, half=False,
             orbit="jittered"),
        # rays from the caller (picking, panoramas, lens models): an odd number of them
        dict(name="rays-100k-401x301", kind="rays", n=100_000, width=401, height=301, degree=2, half=False,
             orbit="plain"),
        # the batched form: 16 uneven views of a 3M scene
        dict(name="batch-3m-16-views", kind="batch", n=3_000_000, width=1920, height=1080, degree=3, half=False,
             views=16),
        # gradients of a small scene for a caller's own optimiser
        dict(name="grad-1k-128x128", kind="grad", n=1000, width=128, height=128, degree=3, half=False, orbit="plain"),
        # early training: odd sizes, low SH degree, jittered pose
        dict(name="train-301k-799x533-deg1", kind="train", n=301_007, width=799, height=533, degree=1, half=False,
             orbit="jittered"),
        # a dense initialisation at the usual training resolution
        dict(name="train-1m-1600x1040", kind="train", n=1_000_000, width=1600, height=1040, degree=3, half=False,
             orbit="jittered"),
        # the headline: a train step at 3M Gaussians and 1080p
        dict(name="train-3m-1080p", kind="train", n=3_000_000, width=1920, height=1080, degree=3, half=False,
             orbit="plain"),
        # the optimiser and the refit by themselves
        dict(name="optim-1m", kind="optim", n=1_000_003, width=64, height=64, degree=3, half=False, orbit="plain"),
        # a full build after pruning
        dict(name="rebuild-2m", kind="rebuild", n=2_000_001, width=64, height=64, degree=0, half=True, orbit="plain"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "display", "rays", "batch", "train", "train", "train", "grad", "optim",
                       "rebuild"])
    most = dict(render=3_000_000, display=6_000_000, rays=100_000, batch=3_000_000, train=3_000_000, grad=300_000,
                optim=3_000_000, rebuild=3_000_000)[kind]
    least = dict(batch=50_000, optim=1000, rebuild=1000).get(kind, 64)
    n = _log_uniform(rng, least, most)
    if kind in ("optim", "rebuild"):
        width = height = 64
    else:
        pixels = {"render": 2_073_600, "display": 8_294_400, "rays": 120_701, "batch": 2_073_600,
                  "train": 2_073_600, "grad": 640 * 480}[kind]
        # the aspect ratio first, then the pixels it leaves room for
        aspect = rng.choice([1.0, 4 / 3, 1.5, 16 / 9, 0.75, 2.3])
        p = _log_uniform(rng, 64 * 64, pixels)
        width = max(16, int(math.sqrt(p * aspect)) - rng.choice([0, 0, 1, 3, 7]))
        height = max(16, min(int(p / width), pixels // width))
    case = dict(kind=kind, n=n, width=width, height=height, degree=rng.choice([0, 1, 2, 3, 3, 3]), half=False,
                orbit=rng.choice(["plain", "jittered"]))
    if kind == "render":
        case["half"] = rng.random() < 0.5
    if kind == "batch":
        case["views"] = rng.randint(2, 16)
    return case


# ------------------------------------------------------------------------------------------------ scenes

def _scene(n, seed):
    """Gaussian parameters on the GPU (the distributions of gray_gb300.synthetic)."""
    gen = torch.Generator(device="cuda").manual_seed(1000 + seed)

    def normal(*shape):
        return torch.randn(*shape, device="cuda", generator=gen)

    def uniform(lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, device="cuda", generator=gen)

    if n < BOX_BELOW:
        mean = uniform(-1.0, 1.0, n, 3)
        log_scale = -3.0 + 0.3 * normal(n, 3)
    else:
        k = 200
        sig = uniform(0.05, 0.5, k, 3)
        dirs = torch.nn.functional.normalize(normal(k, 3), dim=1)
        centre = dirs * ((10.0 - 2.0 * sig.amax(1)) * uniform(0.0, 1.0, k) ** (1.0 / 3.0))[:, None]
        rot = _rotation_matrix(torch.nn.functional.normalize(normal(k, 4), dim=1))
        member = torch.randint(0, k, (n,), device="cuda", generator=gen)
        mean = centre[member] + (rot[member] @ (normal(n, 3) * sig[member])[:, :, None])[:, :, 0]
        log_scale = -4.5 + 0.5 * normal(n, 3)
    return dict(mean=mean, rotation=torch.nn.functional.normalize(normal(n, 4), dim=1), scale=log_scale,
                opacity=normal(n, 1), sh_coeffs_dc=0.5 + 0.2 * normal(n, 1, 3), sh_coeffs_rest=0.05 * normal(n, 15, 3))


def _rotation_matrix(q):
    q = q / q.norm(dim=-1, keepdim=True)
    r, x, y, z = q.unbind(-1)
    return torch.stack([
        torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - r * z), 2 * (x * z + r * y)], -1),
        torch.stack([2 * (x * y + r * z), 1 - 2 * (x * x + z * z), 2 * (y * z - r * x)], -1),
        torch.stack([2 * (x * z - r * y), 2 * (y * z + r * x), 1 - 2 * (x * x + y * y)], -1)], -2)


def _camera(case, seed, width=None, height=None, k=0) -> CameraInfo:
    rng = np.random.default_rng(77 + 100 * seed + k)
    width, height = width or case["width"], height or case["height"]
    if case["n"] < BOX_BELOW:
        a = rng.uniform(0.0, 2.0 * math.pi)
        fov_y = 2.0 * math.atan(0.5)
        return look_at((4.0 * math.cos(a), 4.0 * math.sin(a), 0.5), (0, 0, 0), (0, 0, 1), fov_y, width, height)
    jitter = (0.0, 0.0)
    if case.get("orbit") == "jittered":
        jitter = tuple(rng.uniform(-math.radians(15), math.radians(15), 2))
    return synthetic.orbit_camera(rng.uniform(0.0, 2.0 * math.pi), width, height, jitter_rad=jitter, uid=k)


def _fill(g, scene, degree):
    with torch.no_grad():
        for name in PARAMS:
            getattr(g, name).copy_(scene[name])
        g.current_sh_degree.fill_(degree)


def _pool(case):
    # hit-list words: far more than the scenes composite per pixel (about 10 hits of a 3M scene)
    return 40 * case["width"] * case["height"] + 1_000_000


def _module(case, scene, half=False):
    cfg = gray.RaytracerConfig(ppll_backward_size=_pool(case), lr_mean_init=LATE_RATES["mean"],
                               lr_rotation_init=LATE_RATES["rotation"], lr_scale_init=LATE_RATES["scale"],
                               lr_opacity_init=LATE_RATES["opacity"], lr_sh_dc_init=LATE_RATES["sh_dc"],
                               lr_sh_rest=LATE_RATES["sh_rest"])
    rt = gray.Raytracer(cfg, case["n"], case["width"], case["height"], inference_only=half)
    _fill(rt.cuda_module.get_gaussians(), scene, case["degree"])
    rt.cuda_module.rebuild_bvh()
    return rt


def _tracer(case, scene, width, height, degree=3, training=False):
    rt = classes.Raytracer(width, height, case["n"], 3, 1, _pool(case) if training else 1, inference_only=not training,
                           inference_sh_fp16=False)
    cfg = rt.get_config()
    cfg.alpha_threshold.fill_(ALPHA_MIN)
    cfg.t_threshold.fill_(T_MIN)
    _fill(rt.get_gaussians(), scene, degree)
    rt.rebuild_bvh()
    return rt


def _set_camera(rt, cam):
    c = rt.get_camera()
    c.znear.fill_(0.0)
    c.zfar.fill_(99999.9)
    c.vertical_fov_radians.fill_(float(cam.fov_y))
    c.set_pose(cam.origin_cuda(), cam.rotation_c2w_blender_cuda())


def _target(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(5000 + seed)
    return torch.rand(3, case["height"], case["width"], device="cuda", generator=gen)


def _batch_views(case, seed):
    rng = np.random.default_rng(4000 + seed)
    sizes = [(max(16, case["width"] * a // b), max(16, case["height"] * a // b)) for a, b in
             ((1, 3), (2, 3), (5, 6), (1, 1))]
    pose = dict(case, orbit="jittered")
    # the resolutions are the case's own, the poses the seed's
    picks = np.random.default_rng(case["n"] + case["views"]).integers(0, 4, case["views"])
    return [(0, _camera(pose, int(rng.integers(0, 10_000)), *sizes[int(i)], k=j)) for j, i in enumerate(picks)]


# ------------------------------------------------------------------------------------------------ passes

def prepare(case, seed):
    kind = case["kind"]
    scene = _scene(case["n"], seed)
    s = dict(case=case, cam=_camera(case, seed))
    # the camera's tensors are uploaded once, as a training or serving loop keeps them
    s["cam"].origin_cuda(), s["cam"].rotation_c2w_blender_cuda()
    if kind in ("render", "train", "optim"):
        s["rt"] = _module(case, scene, half=case["half"])
        if kind == "train":
            s["target"] = _target(case, seed)
        if kind == "optim":
            _optimiser_state(s["rt"], seed)
    elif kind == "display":
        s["rt"] = _tracer(case, scene, case["width"], case["height"], case["degree"])
    elif kind == "rays":
        rt = s["rt"] = _tracer(case, scene, case["width"], case["height"], case["degree"])
        _set_camera(rt, s["cam"])
        rt.get_config().render_depth.fill_(True)
        rt.get_config().rays_from_python.fill_(True)
        fb = rt.get_framebuffer()
        o, d = _rays64(case, s["cam"])
        fb.ray_origin.copy_(o.reshape(fb.ray_origin.shape))
        fb.ray_direction.copy_(d.reshape(fb.ray_direction.shape))
    elif kind == "batch":
        s["rt"] = _tracer(case, scene, 64, 64, case["degree"])
        s["views"] = _batch_views(case, seed)
        s["renderer"] = BatchRenderer([s["rt"]])
        s["renderer"].render(s["views"])  # the plan: autotuned and captured on the first render
    elif kind == "grad":
        s["rt"] = _tracer(case, scene, case["width"], case["height"], case["degree"], training=True)
        s["params"] = [scene[k].clone().requires_grad_() for k in PARAMS]
        gen = torch.Generator(device="cuda").manual_seed(6000 + seed)
        s["upstream"] = torch.randn(3, case["height"], case["width"], device="cuda", generator=gen)
    elif kind == "rebuild":
        s["rt"] = _module(case, scene, half=True).cuda_module
    return s


def _optimiser_state(rt, seed):
    """Gradients of one view (half of the Gaussians seen) and moments of the steps before."""
    rt.cuda_module.get_config().zero_grads.fill_(False)  # accumulate: the caller clears the gradients
    g = rt.cuda_module.get_gaussians()
    gen = torch.Generator(device="cuda").manual_seed(7000 + seed)
    seen = torch.rand(g.count, device="cuda", generator=gen) < 0.5
    g.was_visible.copy_(seen[:, None])
    for name in PARAMS:
        t = getattr(g, name)
        shape = (-1,) + (1,) * (t.dim() - 1)
        grad = 1e-6 * torch.randn(t.shape, device="cuda", generator=gen)
        getattr(g, "grad_" + name).copy_(grad * seen.reshape(shape))
        getattr(g, "first_moment_" + name).copy_(5e-7 * torch.randn(t.shape, device="cuda", generator=gen))
        getattr(g, "second_moment_" + name).copy_(1e-12 * torch.rand(t.shape, device="cuda", generator=gen))


def _training_state(g):
    out = {}
    for name in PARAMS:
        out[name] = getattr(g, name)
        out["m_" + name] = getattr(g, "first_moment_" + name)
        out["v_" + name] = getattr(g, "second_moment_" + name)
    return out


def run(s):
    kind = s["case"]["kind"]
    if kind == "render":
        with torch.no_grad():
            image = s["rt"](s["cam"])
        return dict(image=image, channels=s["rt"].cuda_module.get_gaussians().channels)
    if kind == "display":
        rt = s["rt"]
        _set_camera(rt, s["cam"])
        with torch.no_grad():
            rt.forward_pass_display()
        return dict(image=rt.get_framebuffer().output_channels, channels=rt.get_gaussians().channels)
    if kind == "rays":
        rt = s["rt"]
        with torch.no_grad():
            rt.forward_pass()
        fb = rt.get_framebuffer()
        return dict(image=fb.output_channels, depth=fb.output_depth)
    if kind == "batch":
        return s["renderer"].render(s["views"])
    if kind == "train":
        rt = s["rt"]
        image = rt(s["cam"])
        rt.backward((image - s["target"]).abs().mean())
        rt.step()
        return dict(_training_state(rt.cuda_module.get_gaussians()), image=image.detach())
    if kind == "grad":
        mean, rotation, scale, opacity, dc, rest = s["params"]
        image = gray_autograd.render(s["rt"], s["cam"], mean, rotation, scale, opacity, sh_dc=dc, sh_rest=rest)
        grads = torch.autograd.grad(image, s["params"], s["upstream"])
        return dict(zip(PARAMS, grads), image=image.detach())
    if kind == "optim":
        s["rt"].step()
        return _training_state(s["rt"].cuda_module.get_gaussians())
    if kind == "rebuild":
        s["rt"].rebuild_bvh()
        ws = s["rt"].scene_workspace()
        return dict(order=ws.order, codes=ws.codes, nodes=ws.nodes.view(torch.int32), root=ws.root_box)
    raise ValueError(kind)


def work(case):
    n, kind = case["n"], case["kind"]
    sh = 3 * (case["degree"] + 1) ** 2
    pixels = case["width"] * case["height"]
    # hits of a ray: about 24 per million Gaussians of the clustered scene, a handful of the box scene;
    # a hit costs about 90 operations (object-space ray, response, transmittance and colour sums)
    hits = max(2.0, 24e-6 * n) if n >= BOX_BELOW else 0.004 * n
    # what a view reads per Gaussian: its transform (48 B), opacity, mean and coefficients, and writes:
    # its colour
    view = n * (48 + 4 + 12 + sh * (2 if case["half"] else 4) + 12)
    trace = 90.0 * hits * pixels + 8.0 * sh * n
    step = n * 4 * 59 * 7 + n * (44 + 128) + 2 * n * 24  # Adam: p, m, v both ways and g; snapshot; boxes
    if kind in ("render", "display"):
        return dict(bytes=view + 12 * pixels, flops=trace)
    if kind == "rays":
        return dict(bytes=view + 40 * pixels, flops=trace)
    if kind == "batch":
        views = _batch_views(case, 0)
        p = sum(c.image_width * c.image_height for _, c in views)
        return dict(bytes=view + 12 * n * (case["views"] - 1) + 12 * p, flops=90.0 * hits * p + 8.0 * sh * n * len(views))
    if kind == "train":
        return dict(bytes=view + n * 4 * 59 + step + 72 * pixels, flops=1.5 * trace + 12.0 * 59 * n)
    if kind == "grad":
        return dict(bytes=2 * view + n * (4 * 59 + 172) + 72 * pixels, flops=1.5 * trace)
    if kind == "optim":
        return dict(bytes=step, flops=12.0 * 59 * n)
    return dict(bytes=n * (44 + 128 + 32 + 64 + 16), flops=100.0 * n)


# ------------------------------------------------------------------------------------------------ 64 bits

def _rays64(case, cam, dtype=torch.float32):
    """Origins and directions of the camera's rays."""
    rot = torch.from_numpy(cam.rotation_c2w_blender().astype(np.float64)).cuda()
    w, h = case["width"], case["height"]
    th = math.tan(float(np.float32(cam.fov_y)) / 2.0)
    y = th * (1.0 - 2.0 * (torch.arange(h, device="cuda", dtype=torch.float64) + 0.5) / h)
    x = (w / h) * th * (2.0 * (torch.arange(w, device="cuda", dtype=torch.float64) + 0.5) / w - 1.0)
    d = x[None, :, None] * rot[:, 0] + y[:, None, None] * rot[:, 1] - rot[:, 2]
    d = (d / d.norm(dim=-1, keepdim=True)).reshape(-1, 3)
    o = torch.from_numpy(np.asarray(cam.origin, np.float32)).cuda().double().expand_as(d)
    return o.to(dtype).contiguous(), d.to(dtype)


def _colours64(p, origin, degree):
    """SH colours with the reference's real basis, degrees 0 to 3."""
    d = p["mean"] - origin
    x, y, z = (d / torch.sqrt((d * d).sum(-1, keepdim=True).clamp(min=1e-20))).unbind(-1)
    pi = math.pi
    basis = []
    if degree > 0:
        c = math.sqrt(3 / (4 * pi))
        basis += [-c * y, c * z, -c * x]
    if degree > 1:
        c = math.sqrt(15 / (4 * pi))
        basis += [c * x * y, -c * y * z, math.sqrt(5 / (16 * pi)) * (2 * z * z - x * x - y * y), -c * x * z,
                  0.5 * c * (x * x - y * y)]
    if degree > 2:
        a, b, c = math.sqrt(35 / (32 * pi)), math.sqrt(105 / (4 * pi)), math.sqrt(21 / (32 * pi))
        basis += [-a * y * (3 * x * x - y * y), b * x * y * z, -c * y * (4 * z * z - x * x - y * y),
                  math.sqrt(7 / (16 * pi)) * z * (2 * z * z - 3 * x * x - 3 * y * y),
                  -c * x * (4 * z * z - x * x - y * y), 0.5 * b * z * (x * x - y * y), -a * x * (x * x - 3 * y * y)]
    col = math.sqrt(1 / (4 * pi)) * p["sh_coeffs_dc"][:, 0] + 0.5
    for k, v in enumerate(basis):
        col = col + v[:, None] * p["sh_coeffs_rest"][:, k]
    return col.clamp(min=0.0)


def _trace64(p, colours, o, d, quantise):
    """Colours and depths of the rays [R,3].  quantise: alphas rounded to 16 bits as the renderer
    composites them (else exact ones, as its backward differentiates them)."""
    op = torch.sigmoid(p["opacity"][:, 0])
    reach = torch.where(op > ALPHA_MIN, (4.0 * torch.log((op / ALPHA_MIN).clamp(min=1.0))) ** 0.25,
                        torch.zeros_like(op)).detach()
    m = _rotation_matrix(p["rotation"]).transpose(-1, -2) * torch.exp(-p["scale"])[:, :, None]
    lo = torch.einsum("nij,rnj->rni", m, o[:, None, :] - p["mean"][None])
    ld = torch.einsum("nij,rj->rni", m, d)
    t = -(lo * ld).sum(-1) / (ld * ld).sum(-1)
    u = lo + t[..., None] * ld
    q = (u * u).sum(-1)
    hit = (t >= 0) & (q <= reach ** 2) & (op > ALPHA_MIN)
    alpha = torch.where(hit, MAX_ALPHA * op * torch.exp(-0.25 * q * q), torch.zeros_like(q))
    dist = t.detach().half().double()
    full = torch.prod(1.0 - alpha, dim=-1)
    order = torch.argsort(torch.where(hit, dist, torch.full_like(dist, math.inf)), dim=-1, stable=True)
    a = torch.gather(alpha, 1, order)
    if quantise:
        a = a.half().double()
    c, dist = colours[order], torch.gather(dist, 1, order)
    after = torch.cumprod(1.0 - a, dim=-1)
    before = torch.cat([torch.ones_like(after[:, :1]), after[:, :-1]], dim=-1)
    taken = (before.detach() >= T_MIN) & (a.detach() > 0) & (dist > 0)
    w = torch.where(taken, before * a, torch.zeros_like(a))
    left = torch.prod(torch.where(taken, 1.0 - a, torch.ones_like(a)), dim=-1)
    skipped = torch.where(taken, torch.zeros_like(a), a).detach()
    total = skipped.sum(-1, keepdim=True)
    rest = torch.where(total > 0, (skipped[..., None] * c).sum(1).detach() / total.clamp(min=1e-300),
                       torch.zeros_like(c[:, 0]))
    depth = torch.where(taken, w * dist, torch.zeros_like(w)).sum(-1) / (1.0 - left).clamp(min=1e-12)
    return (w[..., None] * c).sum(1) + (left - full)[:, None] * rest, depth


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind in ("batch", "train", "rebuild"):
        return None
    if kind == "rays":
        return None
    scene = _scene(n, seed)
    if kind == "optim":
        return _exact_optim(case, scene, seed)
    cam = _camera(case, seed)
    if case["half"]:
        scene = {k: v.half() if k.startswith("sh_") else v for k, v in scene.items()}
    p = {k: v.double() for k, v in scene.items()}
    origin = torch.from_numpy(np.asarray(cam.origin, np.float32)).cuda().double()
    w, h = case["width"], case["height"]
    small = n * w * h <= 70_000_000
    chunk = max(16, 4_000_000 // n)
    if kind == "grad" and not small:
        return None
    if kind == "grad":
        for v in p.values():
            v.requires_grad_()
    colours = _colours64(p, origin, case["degree"])
    image = None
    if small:
        o, d = _rays64(case, cam, torch.float64)
        with torch.no_grad():
            image = torch.cat([_trace64(p, colours, o[i:i + chunk], d[i:i + chunk], True)[0]
                               for i in range(0, w * h, chunk)]).reshape(h, w, 3)
    if kind == "display":
        return dict(image=image, channels=colours)
    if image is not None:
        image = image.permute(2, 0, 1)
    if kind == "render":
        return dict(image=image, channels=colours)
    gen = torch.Generator(device="cuda").manual_seed(6000 + seed)
    up = torch.randn(3, h, w, device="cuda", generator=gen).double().permute(1, 2, 0).reshape(-1, 3)
    held = colours.detach().requires_grad_()
    for i in range(0, w * h, chunk):
        img = _trace64(p, held, o[i:i + chunk], d[i:i + chunk], False)[0]
        (img * up[i:i + chunk]).sum().backward()
    if case["degree"] == 0:
        p["sh_coeffs_rest"].grad = torch.zeros_like(p["sh_coeffs_rest"])
    colours.backward(held.grad)
    return dict({k: p[k].grad for k in PARAMS}, image=image)


def _exact_optim(case, scene, seed):
    n = case["n"]
    gen = torch.Generator(device="cuda").manual_seed(7000 + seed)
    seen = torch.rand(n, device="cuda", generator=gen) < 0.5
    rate = dict(zip(PARAMS, (LATE_RATES[k] for k in ("mean", "rotation", "scale", "opacity", "sh_dc", "sh_rest"))))
    b1, b2 = float(np.float32(0.9)), float(np.float32(0.999))
    out = {}
    for name in PARAMS:
        t = scene[name]
        grad = (1e-6 * torch.randn(t.shape, device="cuda", generator=gen)
                * seen.reshape((-1,) + (1,) * (t.dim() - 1))).double()
        m = (5e-7 * torch.randn(t.shape, device="cuda", generator=gen)).double()
        v = (1e-12 * torch.rand(t.shape, device="cuda", generator=gen)).double()
        m = b1 * m + (1 - b1) * grad
        v = b2 * v + (1 - b2) * grad * grad
        # the first step: the bias corrections take the exponent step + 1
        lr = float(np.float32(rate[name]))
        p = t.double() - lr * (m / (1 - b1 ** 2)) / ((v / (1 - b2 ** 2)).sqrt() + 1e-15)
        out[name], out["m_" + name], out["v_" + name] = p, m, v
    return out
