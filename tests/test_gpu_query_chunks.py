"""Host ray queries are split into chunks over several workers: a call gives what
the same rays give in small calls, at every number of rays where the split changes,
and from several threads at once (GPU). Closest-hit calls are split from 131,072
rays on, and a miss of theirs is zero in every output.
"""

import threading

import numpy as np
import pytest

import albedo_b200 as ab
from albedo_b200 import scenes

pytestmark = pytest.mark.gpu

SMALL = 8192  # run whole


@pytest.fixture(scope="module")
def scene(tmp_path_factory):
    return ab.Scene.load(scenes.trefoil_scene(tmp_path_factory.mktemp("chunks")))


def rays_of(count, seed):
    rng = np.random.default_rng(seed)
    origins = rng.uniform([-3, 0.05, -3.5], [3, 4, 4], size=(count, 3))
    directions = rng.normal(size=(count, 3))
    return np.concatenate([origins, directions], axis=1).astype(np.float32)


def in_pieces(query, count):
    parts = [query(slice(i, min(i + SMALL, count))) for i in range(0, count, SMALL)]
    if isinstance(parts[0], dict):
        return {k: np.concatenate([p[k] for p in parts]) for k in parts[0]}
    return np.concatenate(parts)


@pytest.mark.parametrize("count", [1, 16385, 131071, 131072, 131073, 8 * 32768, 8 * 32768 + 1, 300007])
@pytest.mark.parametrize("geometry", [False, True])
def test_closest_hits_equal_those_of_small_calls(scene, count, geometry):
    rays = rays_of(count, count)
    whole = scene.intersect(rays, t_max=3.0, geometry=geometry)
    parts = in_pieces(lambda s: scene.intersect(rays[s], t_max=3.0, geometry=geometry), count)
    np.testing.assert_array_equal(whole["hit"], parts["hit"])
    hits = whole["hit"] != 0
    for name, values in whole.items():
        np.testing.assert_array_equal(values[hits], parts[name][hits], err_msg=name)
        if count >= 131072:
            assert not np.any(values[~hits]), name


@pytest.mark.parametrize("count", [1, 16385, 8 * 32768 + 1])
def test_occlusion_equals_that_of_small_calls(scene, count):
    rays = rays_of(count, count)
    t_max = np.random.default_rng(1).uniform(0.1, 3.0, count).astype(np.float32)
    np.testing.assert_array_equal(scene.occluded(rays, t_max),
                                  in_pieces(lambda s: scene.occluded(rays[s], t_max[s]), count))


def test_queries_from_several_threads(scene):
    work = [rays_of(131_072 + 9000 * k, k) for k in range(6)]
    alone = [scene.intersect(r) for r in work]
    together = [None] * len(work)

    def run(k):
        for _ in range(3):
            together[k] = scene.intersect(work[k])

    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(work))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(alone, together):
        for name in a:
            np.testing.assert_array_equal(a[name], b[name], err_msg=name)


def test_no_rays(scene):
    assert len(scene.intersect(np.zeros((0, 6), np.float32))["hit"]) == 0
    assert len(scene.occluded(np.zeros((0, 6), np.float32), np.zeros(0, np.float32))) == 0
