"""The values set_view takes and refuses are those that fill_ takes and refuses.  Needs a GB300."""
import math

import numpy as np
import pytest
import torch

import gray_gb300 as gray
from gray_gb300 import classes, synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda(gray_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _pose():
    return torch.tensor([0.5, -2.0, 3.0], device="cuda"), torch.eye(3, device="cuda")


def _values(rt):
    c = rt.get_camera()
    return [t.item() for t in (c.vertical_fov_radians, c.znear, c.zfar)]


@pytest.mark.parametrize("kind", ["tensor", "host tensor", "numpy", "int", "inf"])
def test_set_view_takes_what_fill_takes(kind):
    rt = classes.Raytracer(16, 8, 4, 0, 1, 1000)
    given = {"tensor": [torch.tensor(v, device="cuda") for v in (0.75, 0.25, 80.0)],
             "host tensor": [torch.tensor(v, dtype=torch.float64) for v in (0.75, 0.25, 80.0)],
             "numpy": [np.float32(0.75), np.float64(0.25), np.float32(80.0)], "int": [1, 0, 80],
             "inf": [0.75, -math.inf, math.inf]}[kind]
    rt.set_view(*_pose(), *given)
    assert _values(rt) == [float(v) for v in given]


def test_views_by_device_values_are_captured():
    """znear, zfar and the field of view as device tensors: no wait for them, so a graph takes the call."""
    rt = gray.Raytracer(gray.RaytracerConfig(ppll_backward_size=1), 64, 16, 8, inference_only=True)
    sc = synthetic.small_scene(n=64)
    with torch.no_grad():
        for name in ("mean", "rotation", "scale", "opacity"):
            getattr(rt.cuda_module.get_gaussians(), name).copy_(torch.from_numpy(getattr(sc, name)))
    rt.cuda_module.rebuild_bvh()
    cam = synthetic.look_at((0.0, -3.0, 0.4), (0, 0, 0), (0, 0, 1), 0.6, 16, 8)
    near, far = torch.tensor(0.5, device="cuda"), torch.tensor(50.0, device="cuda")
    cam.fov_y = torch.tensor(0.625, device="cuda")
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.no_grad(), torch.cuda.stream(stream):
        rt(cam, znear=near, zfar=far)
        stream.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            image = rt(cam, znear=near, zfar=far)
    near.fill_(1.0)
    graph.replay()
    torch.cuda.synchronize()
    assert _values(rt.cuda_module) == [0.625, 1.0, 50.0] and bool(torch.isfinite(image).all())


@pytest.mark.parametrize("which", [0, 1, 2])
def test_set_view_refuses_what_fill_refuses(which):
    rt = classes.Raytracer(16, 8, 4, 0, 1, 1000)
    values = [0.75, 0.25, 80.0]
    values[which] = 1e39
    with pytest.raises(RuntimeError):
        rt.get_camera().znear.fill_(1e39)
    with pytest.raises(RuntimeError):
        rt.set_view(*_pose(), *values)
