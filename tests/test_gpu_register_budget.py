"""The megakernel's register budget is chosen by the size of the image and what
queries of the scene's meshes cost: at the sizes where the choice changes, an untuned scene's image is
the one both budgets give, bit for bit (GPU).
"""

import numpy as np
import pytest
import torch

import albedo_b200 as ab
from albedo_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def make(tmp_path_factory):
    directory = tmp_path_factory.mktemp("budget")
    paths = {"room": scenes.room_scene(directory), "soup": scenes.soup_scene(directory, count=100_000)}
    return lambda name: ab.Scene.load(paths[name])


def render(scene, job):
    acc = torch.zeros((job.width * job.height, 4), dtype=torch.float64, device="cuda")
    ab.render_device(scene, job, acc.data_ptr())
    torch.cuda.synchronize()
    scene.check()
    return acc.cpu().numpy()


# Warps of 32 pixels, 12 per SM: 20 such waves at 960 rows of 8 pixels an SM, 6 at 288.
@pytest.mark.parametrize("name,rows", [("room", 959), ("room", 960), ("soup", 287), ("soup", 288)])
@pytest.mark.parametrize("accumulation", [ab.ACCUMULATE_FP64, ab.ACCUMULATE_KAHAN_FP32])
def test_both_budgets_give_the_chosen_ones_image(make, name, rows, accumulation):
    scene = make(name)
    width = 8 * torch.cuda.get_device_properties(0).multi_processor_count
    job = ab.RenderJob(width, rows, samples_per_axis=1, seed=5, max_depth=5, accumulation=accumulation)
    chosen = render(scene, job)
    for blocks in (3, 4):
        ab.set_tuning(scene, tile_width=16, blocks_per_sm=blocks, inline_traversal=0)
        np.testing.assert_array_equal(render(scene, job).view(np.int64), chosen.view(np.int64))
