"""A megakernel shape that was read can be set again: a scene without a shape of its
own stays without one, and one with a shape keeps it (host)."""

from __future__ import annotations

import pytest

import albedo_b200 as ab


def test_a_scene_without_a_shape_stays_without_one():
    scene = ab.Scene.create()
    fresh = ab.tuning(scene)
    assert fresh["evaluations"] == -1 and (fresh["tile_width"], fresh["blocks_per_sm"]) == (16, 3)
    ab.set_tuning(scene, **fresh)
    assert ab.tuning(scene) == fresh
    # Pinned to the same values it has one, until what was read first is set again.
    ab.set_tuning(scene, tile_width=16, blocks_per_sm=3, inline_traversal=0)
    assert ab.tuning(scene)["evaluations"] == 0
    ab.set_tuning(scene, **fresh)
    assert ab.tuning(scene) == fresh


@pytest.mark.parametrize("blocks,inline", [(3, 0), (3, 2), (4, 1)])
def test_a_scenes_own_shape_is_kept(blocks, inline):
    scene = ab.Scene.create()
    ab.set_tuning(scene, tile_width=8, blocks_per_sm=blocks, inline_traversal=inline)
    own = ab.tuning(scene)
    assert own["evaluations"] == 0
    ab.set_tuning(scene, tile_width=32, blocks_per_sm=3)
    ab.set_tuning(scene, **own)
    assert ab.tuning(scene) == own


def test_unknown_fields_and_shapes_are_refused():
    scene = ab.Scene.create()
    for shape in ({"tiles": 8}, {"tile_width": 12, "blocks_per_sm": 3}, {"tile_width": 16, "blocks_per_sm": 0}):
        with pytest.raises(ValueError):
            ab.set_tuning(scene, **shape)
