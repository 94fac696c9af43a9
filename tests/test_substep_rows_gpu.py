"""The substep kernel's register variants (needs a B200).

A batch's 256-thread class runs the one-block-an-SM variant up to two
worlds an SM and the denser one beyond; a single world always runs the
first.  The same world stepped alone, in a batch below the line and in one
above it must hash the same: stacks, joints with motors and limits,
restitution, terrain contacts.
"""
import pytest

from conftest import cuda_available
from maul3d_b200.abi import (SCENE_BOUNCE, SCENE_BOX_PYRAMID, SCENE_PLANK, SCENE_TOWERS,
                             SCENE_UNEVEN)

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

DT = 1.0 / 60.0


@pytest.mark.parametrize("spec", [(SCENE_BOX_PYRAMID, 0, 20), (SCENE_UNEVEN, 3, 200),
                                  (SCENE_TOWERS, 4, 20), (SCENE_PLANK, 5, 200),
                                  (SCENE_BOUNCE, 6, 220)])
@pytest.mark.parametrize("count", [296, 297])
def test_batches_about_the_line_equal_one_world(m3, spec, count):
    alone = m3.World.scene(*spec)
    worlds = [m3.World.scene(*spec) for _ in range(count)]
    try:
        for _ in range(4):
            alone.step(DT, 4, 5)
            m3.step_worlds(worlds, DT, 4, 5)
            expected = alone.hash()
            hashes = [int(x) for x in m3.hash_worlds(worlds)]
            assert hashes == [expected] * count
    finally:
        alone.destroy()
        for w in worlds:
            w.destroy()
