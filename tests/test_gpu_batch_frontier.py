"""A batch group's frontier holds as many nodes as a tile's of the plain forward.  Needs a GB300."""
import numpy as np
import pytest
import torch

from gray_gb300 import synthetic
from gray_gb300.batch import BatchRenderer
from tests import gpu_util as G

pytestmark = pytest.mark.gpu


def test_batch_frontiers_of_up_to_160_nodes(gray_lib):
    """Wide groups of a clustered scene reach from a few to some hundred nodes: those with 158 to 160 start
    at their frontier too, none holds more, and the pixels are the plain forward's."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sc = synthetic.clustered_scene(200_000, seed=3)
    rt = G.make_tracer(64, 48, sc.mean, sc.rotation, sc.scale, sc.opacity, inference_only=True,
                       channels=np.random.default_rng(1).uniform(0, 1, (sc.n, 3)).astype(np.float32))
    cams = [synthetic.orbit_camera(0.39 * k, 64, 48) for k in range(16)]
    br = BatchRenderer([rt], use_graph=False, autotune=False, variant=5, blocks_per_sm=1)
    images = [i.clone() for i in br.render([(0, c) for c in cams])]
    plan = next(iter(br.plans.values()))
    words = int(gray_lib.gray_frontier_words())
    counts = plan.frontier.view(-1, words)[:plan.total_groups, 0].cpu().numpy()
    counts = counts[counts >= 0]
    assert (counts > 157).any() and counts.max() <= 160, np.sort(counts)[-10:]
    for c, image in zip(cams, images):
        rt.set_view(c.origin_cuda(), c.rotation_c2w_blender_cuda(), c.fov_y, 0.0, 99999.9)
        rt.forward_pass_display()
        assert torch.equal(image, rt.get_framebuffer().output_channels.moveaxis(-1, 0))
