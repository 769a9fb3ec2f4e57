"""A miss of a closest-hit query is zero in every output at every number of rays,
whatever the device memory held before (GPU).
"""

import numpy as np
import pytest

import albedo_b200 as ab
from albedo_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(tmp_path_factory):
    return ab.Scene.load(scenes.icosphere_scene(tmp_path_factory.mktemp("misses"), levels=3))


@pytest.mark.parametrize("count", [1, 33, 1000, 16384, 16385, 131071, 131072])
@pytest.mark.parametrize("geometry", [False, True])
def test_misses_are_zero(scene, count, geometry):
    down = np.tile(np.array([0, 9, 0, 0, -1, 0], np.float32), (count, 1))
    hits = scene.intersect(down, geometry=geometry)
    assert np.all(hits["hit"] == 1) and np.all(hits["t"] > 0)
    # The same call just after it, of rays that start outside and leave.
    misses = scene.intersect(down * np.array([1, 1, 1, 1, -1, 1], np.float32), geometry=geometry)
    for name, values in misses.items():
        assert not np.any(values), name
    # Every other ray misses.
    mixed = down.copy()
    mixed[::2, 4] = 1
    found = scene.intersect(mixed, geometry=geometry)
    for name, values in found.items():
        assert not np.any(values[::2]), name
        np.testing.assert_array_equal(values[1::2], hits[name][1::2], err_msg=name)
