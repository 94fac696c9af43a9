"""The contact colouring's two forms (needs a B200).

A wide world colours along its constraints' chains over the whole grid, a
world of one block in rounds and then, for chains longer than the rounds, by
one warp.  Both must give the serial walk's colours, so twin worlds stepped
either way keep the same hash and colour count: no row, a few rows, chains
on either side of the round limit, several rows between the same two
bodies, more rows on a body than there are colours.
"""
import pytest

from conftest import cuda_available
from maul3d_b200.abi import (SCENE_BOX_PYRAMID, SCENE_FREEFALL, SCENE_MIXED, SCENE_PLANK,
                             SCENE_RAIN, SCENE_TOWERS, SCENE_UNEVEN)

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

DT = 1.0 / 60.0


@pytest.mark.parametrize("spec,steps", [
    ((SCENE_FREEFALL, 0, 8), 3), ((SCENE_BOX_PYRAMID, 0, 1), 20), ((SCENE_BOX_PYRAMID, 0, 6), 20),
    ((SCENE_BOX_PYRAMID, 0, 12), 20), ((SCENE_BOX_PYRAMID, 0, 55), 12), ((SCENE_UNEVEN, 5, 33), 60),
    ((SCENE_UNEVEN, 9, 1500), 40), ((SCENE_TOWERS, 3, 12), 20), ((SCENE_PLANK, 2, 60), 60),
    ((SCENE_MIXED, 4, 900), 40), ((SCENE_RAIN, 8, 400), 60)])
def test_wide_and_one_block_colours_agree(m3, spec, steps):
    previous = m3.set_wide_min_shapes(0)
    narrow, wide = m3.World.scene(*spec), m3.World.scene(*spec)
    try:
        for step in range(steps):
            for world, threshold in ((narrow, 1 << 30), (wide, 1)):
                m3.set_wide_min_shapes(threshold)
                world.step(DT, 2, 1)
            assert wide.hash() == narrow.hash(), f"step {step + 1}"
            assert m3.counters(wide) == m3.counters(narrow), f"step {step + 1}"
    finally:
        m3.set_wide_min_shapes(previous)
        narrow.destroy()
        wide.destroy()
