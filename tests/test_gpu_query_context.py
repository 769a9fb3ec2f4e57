"""Host ray queries in a CUDA context that the program made itself: the scene's
tables, the workers' buffers and the kernels are all in it, and it stays current in
the caller's thread (GPU).
"""

import ctypes
from contextlib import contextmanager

import numpy as np
import pytest
import torch

import albedo_b200 as ab
from albedo_b200 import scenes

pytestmark = pytest.mark.gpu


@contextmanager
def own_context():
    driver = ctypes.CDLL("libcuda.so.1")
    context, popped = ctypes.c_void_p(), ctypes.c_void_p()
    assert driver.cuCtxCreate_v2(ctypes.byref(context), 0, 0) == 0
    try:
        yield driver, context.value
    finally:
        assert driver.cuCtxPopCurrent_v2(ctypes.byref(popped)) == 0 and popped.value == context.value
        assert driver.cuCtxDestroy_v2(context) == 0


def test_the_callers_context_is_used_and_stays(tmp_path):
    path = scenes.icosphere_scene(tmp_path, levels=3)
    rng = np.random.default_rng(5)
    count = 100_003
    rays = np.concatenate([rng.uniform([-3, 0.05, -3.5], [3, 4, 4], (count, 3)), rng.normal(size=(count, 3))], axis=1)
    rays = rays.astype(np.float32)
    far = np.full(count, 2.0, np.float32)
    torch.cuda.synchronize()  # the primary context is there, and current
    scene = ab.Scene.load(path)
    hits, blocked = scene.intersect(rays, geometry=True), scene.occluded(rays, far)
    with own_context() as (driver, context):
        own = ab.Scene.load(path)
        for _ in range(2):
            found, shadow = own.intersect(rays, geometry=True), own.occluded(rays, far)
            now = ctypes.c_void_p()
            assert driver.cuCtxGetCurrent(ctypes.byref(now)) == 0 and now.value == context
            for name, values in found.items():
                np.testing.assert_array_equal(values, hits[name], err_msg=name)
            np.testing.assert_array_equal(shadow, blocked)
        own.close()
    again = scene.intersect(rays, geometry=True)
    for name, values in again.items():
        np.testing.assert_array_equal(values, hits[name], err_msg=name)
