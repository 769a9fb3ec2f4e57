"""Arrays that the host cannot read or write are an error of a ray query, not a
crash; an output that is not wanted may be null, and arrays that a call does not
use may be anything (GPU).
"""

import ctypes

import numpy as np
import pytest
import torch

import albedo_b200 as ab
from albedo_b200 import scenes
from albedo_b200._lib import library

pytestmark = pytest.mark.gpu

DEVICE_ERROR = 5  # include/albedo_b200.h
FLOATS, INTS = ctypes.POINTER(ctypes.c_float), ctypes.POINTER(ctypes.c_int32)


def at(address, kind):
    return ctypes.cast(ctypes.c_void_p(address), kind)


@pytest.fixture(scope="module")
def scene(tmp_path_factory):
    return ab.Scene.load(scenes.room_scene(tmp_path_factory.mktemp("arrays")))


def rays_of(count):
    rays = np.zeros((count, 6), np.float32)
    rays[:, 1], rays[:, 5] = 1.0, -1.0
    return rays


@pytest.mark.parametrize("count", [64, 40_000, 140_000])
def test_arrays_the_host_cannot_touch_are_refused(scene, count):
    rays, far = rays_of(count), np.full(count, 0.5, np.float32)
    on_device = torch.zeros((count, 6), device="cuda").data_ptr()
    good = {"rays": rays.ctypes.data, "far": far.ctypes.data}

    def occluded(**given):
        use = {**good, "out": np.zeros(count, np.int32).ctypes.data, **given}
        return library().albedo_occluded_host(scene.handle, at(use["rays"], FLOATS), at(use["far"], FLOATS), count,
                                              at(use["out"], INTS))

    out = np.zeros(count, np.int32)
    assert occluded(out=out.ctypes.data) == 0
    np.testing.assert_array_equal(out, scene.occluded(rays, far))
    assert occluded(out=None) == 0
    for bad in ({"rays": None}, {"far": None}, {"rays": on_device}, {"far": on_device}, {"out": on_device}):
        assert occluded(**bad) == DEVICE_ERROR, bad


@pytest.mark.parametrize("count", [64, 140_000])
def test_closest_hits_with_unwanted_and_unused_arrays(scene, count):
    rays = rays_of(count)
    on_device = torch.zeros((count, 3), device="cuda").data_ptr()
    hit, t = np.zeros(count, np.int32), np.zeros(count, np.float32)

    def trace(point=None, normal=None, t_out=t.ctypes.data, rays_in=rays.ctypes.data):
        return library().albedo_trace_host(
            scene.handle, at(rays_in, FLOATS), count, 0.0, float("inf"), at(hit.ctypes.data, INTS), at(t_out, FLOATS),
            None, None, at(point, FLOATS), at(normal, FLOATS), None, None)

    assert trace() == 0
    expected = scene.intersect(rays)
    np.testing.assert_array_equal(hit, expected["hit"])
    np.testing.assert_array_equal(t, expected["t"])
    assert trace(normal=on_device) == 0  # no geometry asked for: not looked at
    point = np.zeros((count, 3), np.float32)
    assert trace(point=point.ctypes.data) == 0
    np.testing.assert_array_equal(point, scene.intersect(rays, geometry=True)["point"])
    for bad in ({"point": on_device}, {"point": point.ctypes.data, "normal": on_device}, {"t_out": on_device},
                {"rays_in": None}, {"rays_in": on_device}):
        assert trace(**bad) == DEVICE_ERROR, bad


def test_no_rays_need_no_arrays(scene):
    assert library().albedo_occluded_host(scene.handle, None, None, 0, None) == 0
    assert library().albedo_trace_host(scene.handle, None, 0, 0.0, 1.0, None, None, None, None, None, None, None,
                                       None) == 0
