"""Renders too small for full warps spread their pixels over more warps; every
pixel's sum is the one it has in a large image (GPU).

A pixel's random stream depends on its place and the image's width alone, so a
list of pixels of a 400x225 frame renders bit for bit what the frame, rendered
with full warps, holds there. The lists' lengths sit on both sides of every
change of the pixels a warp takes: 3 warps per SM for a scene without
triangles, 12 with a mesh (148 SMs).
"""

import numpy as np
import pytest
import torch

import albedo_b200 as ab
from albedo_b200 import scenes

pytestmark = pytest.mark.gpu

WIDTH, HEIGHT = 400, 225


@pytest.fixture(scope="module")
def frames(tmp_path_factory):
    directory = tmp_path_factory.mktemp("small")
    job = ab.RenderJob(WIDTH, HEIGHT, samples_per_axis=2, seed=3, max_depth=6)
    made = {}
    for name, path in [("room", scenes.room_scene(directory / "room")),
                       ("mesh", scenes.icosphere_scene(directory / "mesh", levels=4))]:
        scene = ab.Scene.load(path)
        acc = torch.zeros((WIDTH * HEIGHT, 4), dtype=torch.float64, device="cuda")
        ab.render_device(scene, job, acc.data_ptr())
        torch.cuda.synchronize()
        scene.check()
        made[name] = scene, job, acc.cpu().numpy()
    return made


@pytest.mark.parametrize("name,warps", [("room", 444), ("mesh", 1776)])
@pytest.mark.parametrize("lanes", [1, 2, 4, 8, 16, 32])
def test_spread_pixels_equal_the_full_frame(frames, name, warps, lanes):
    scene, job, frame = frames[name]
    order = np.random.default_rng(lanes).permutation(WIDTH * HEIGHT)
    for count in {1, warps * lanes // 2 + 1, warps * lanes}:
        chosen = order[:count]
        pixels = np.stack([chosen % WIDTH, chosen // WIDTH], axis=1)
        acc = ab.render_pixels(scene, job, pixels)
        for k, field in enumerate(("r", "g", "b")):
            np.testing.assert_array_equal(acc[field], frame[chosen, k])
        assert np.all(acc["count"] == 4)


@pytest.mark.parametrize("width,height", [(1, 1), (3, 5), (17, 9), (29, 31), (64, 36), (97, 53), (131, 61)])
def test_small_images_cover_every_pixel_once(frames, width, height):
    scene, _, _ = frames["mesh"]
    job = ab.RenderJob(width, height, samples_per_axis=3, seed=5, max_depth=4)
    image = ab.PixelBuffer(width, height)
    ab.render_image(scene, job, image)
    assert np.all(image.pixels["count"] == 9)
    listed = ab.render_pixels(scene, job, np.stack(np.divmod(np.arange(width * height), width)[::-1], axis=1))
    np.testing.assert_array_equal(listed, image.pixels)
