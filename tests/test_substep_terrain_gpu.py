"""The substep kernel's register variants on heightfield contacts (needs a
B200).

A batch's 256-thread class runs the one-block-an-SM variant up to two
worlds an SM and the denser one beyond.  Worlds of that class (161 to 768
slots) on a heightfield, stepped alone and in batches on either side of
the device's own line, must hash the same.
"""
import pytest

from conftest import cuda_available
from maul3d_b200.abi import SCENE_TERRAIN

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

DT = 1.0 / 60.0


@pytest.mark.parametrize("size", [170, 300])
@pytest.mark.parametrize("beyond", [0, 1])
def test_terrain_batches_about_the_line_equal_one_world(m3, size, beyond):
    import torch
    count = 2 * torch.cuda.get_device_properties(0).multi_processor_count + beyond
    alone = m3.World.scene(SCENE_TERRAIN, 7, size)
    worlds = [m3.World.scene(SCENE_TERRAIN, 7, size) for _ in range(count)]
    try:
        assert 161 <= alone.body_count() <= 768  # a shape a body
        for steps in (4, 26):
            alone.step(DT, 4, steps)
            m3.step_worlds(worlds, DT, 4, steps)
            assert [int(x) for x in m3.hash_worlds(worlds)] == [alone.hash()] * count
    finally:
        alone.destroy()
        for w in worlds:
            w.destroy()
