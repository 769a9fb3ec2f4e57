"""Host ray queries read their arrays after the work that the default stream held
when the call was made (GPU): pinned rays that a copy, queued behind other work on
the default stream or on a stream ordered with it, is still to fill.
"""

import ctypes

import numpy as np
import pytest
import torch

import albedo_b200 as ab
from albedo_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(tmp_path_factory):
    return ab.Scene.load(scenes.icosphere_scene(tmp_path_factory.mktemp("order"), levels=3))


@pytest.fixture(scope="module")
def blocking_stream():
    """A stream that orders itself with the default one (torch's own do not)."""
    driver = ctypes.CDLL("libcuda.so.1")
    torch.zeros(1, device="cuda")
    stream = ctypes.c_void_p()
    assert driver.cuStreamCreate(ctypes.byref(stream), 0) == 0
    yield torch.cuda.ExternalStream(stream.value)
    torch.cuda.synchronize()
    assert driver.cuStreamDestroy_v2(stream) == 0


@pytest.mark.parametrize("count", [1, 1000, 131_072])
@pytest.mark.parametrize("where", ["default", "blocking"])
def test_pinned_rays_filled_by_a_queued_copy(scene, blocking_stream, count, where):
    down = torch.tensor([0, 9, 0, 0, -1, 0], dtype=torch.float32).repeat(count, 1)
    up = down * torch.tensor([1, 1, 1, 1, -1, 1])
    on_device = down.cuda()
    pinned = up.clone().pin_memory()
    torch.cuda.synchronize()
    stream = torch.cuda.default_stream() if where == "default" else blocking_stream
    far = np.full(count, 100.0, np.float32)
    for query in (lambda rays: scene.intersect(rays)["hit"], lambda rays: scene.occluded(rays, far)):
        pinned.copy_(up)
        with torch.cuda.stream(stream):
            torch.cuda._sleep(100_000_000)  # about 50 ms
            pinned.copy_(on_device, non_blocking=True)
        assert np.all(query(pinned.numpy()) == 1)
        torch.cuda.synchronize()
