"""set_view against the holders' own setters, and the forward that stores its gradient mode.  Needs a GB300."""
import pytest
import torch

from gray_gb300 import classes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["plain", "double", "transposed", "host"])
@pytest.mark.parametrize("n", [0, 1, 63, 64, 65, 200])
def test_set_view_and_forward_mode(gray_lib, kind, n):
    """Contiguous float32 device tensors go through one launch, others through set_pose: the camera
    holds the same values either way; forward_pass stores torch's gradient mode with or without Gaussians."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rt = classes.Raytracer(16, 8, max(n, 1), 0, 1, 1000)
    if n == 0:
        rt.resize(0)
    rt.rebuild_bvh()
    origin = torch.tensor([0.5, -2.0, 3.0], device="cuda")
    rot = torch.linalg.qr(torch.randn(3, 3, generator=torch.Generator().manual_seed(n)))[0].cuda()
    given = dict(plain=(origin, rot), double=(origin.double(), rot.double()), transposed=(origin, rot.t()),
                 host=(origin.cpu(), rot.cpu()))[kind]
    rt.get_config().rays_from_python.fill_(True)
    rt.set_view(*given, 0.75, 0.25, 80.0)
    c, r = rt.get_camera(), rot.t() if kind == "transposed" else rot
    assert torch.equal(c.origin, origin) and torch.equal(c.rotation_c2w, r) and torch.equal(c.rotation_w2c, r.t())
    assert c.vertical_fov_radians.item() == 0.75 and c.znear.item() == 0.25 and c.zfar.item() == 80.0
    assert not rt.get_config().rays_from_python.item()
    for mode in (True, False, True):
        with torch.set_grad_enabled(mode):
            rt.forward_pass()
        assert bool(rt.get_metadata().grads_enabled.item()) == mode
    rt.check_status()
