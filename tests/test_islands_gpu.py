"""A wide world's substep loop by islands (needs a B200).

A wide world whose islands fit the blocks' groups runs each group's substep
loop in a block of its own; a world of one block (not wide) runs the
per-world kernels.  Twin worlds step both ways and every step's hash and
the snapshot at the end must be the same: towers of breakable joints,
revolute chains, restitution, the overflow colour inside an island, one
island holding every row (too large for a group: the grid's levels), a
kinematic mover (the grid's levels), sleeping islands, a world without a
single row.
"""
import ctypes as C

import pytest

from conftest import cuda_available
from maul3d_b200 import abi
from maul3d_b200.abi import (SCENE_BOUNCE, SCENE_BOX_PYRAMID, SCENE_CITY, SCENE_FREEFALL,
                             SCENE_MIXED, SCENE_PLANK, SCENE_RAIN, SCENE_TERRAIN, SCENE_TOWERS,
                             SCENE_UNEVEN)

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

DT = 1.0 / 60.0


def _twins(m3, make, substeps, steps, between=None):
    previous = m3.set_wide_min_shapes(0)
    narrow, wide = make(), make()
    try:
        for step in range(steps):
            for w, threshold in ((narrow, 1 << 30), (wide, 1)):
                if between is not None:
                    between(w, step)
                m3.set_wide_min_shapes(threshold)
                w.step(DT, substeps, 1)
            assert wide.hash() == narrow.hash(), f"step {step + 1}"
        assert m3.snapshot(wide) == m3.snapshot(narrow)
    finally:
        m3.set_wide_min_shapes(previous)
        narrow.destroy()
        wide.destroy()


@pytest.mark.parametrize("spec,substeps,steps", [
    ((SCENE_FREEFALL, 0, 40), 4, 5), ((SCENE_UNEVEN, 7, 400), 4, 60),
    ((SCENE_TOWERS, 8, 9), 4, 90), ((SCENE_CITY, 9, 3), 8, 45), ((SCENE_PLANK, 5, 40), 4, 60),
    ((SCENE_BOUNCE, 6, 150), 4, 120), ((SCENE_BOX_PYRAMID, 0, 40), 4, 30),
    ((SCENE_TERRAIN, 3, 1500), 2, 60), ((SCENE_RAIN, 3, 600), 1, 60),
    ((SCENE_MIXED, 4, 2500), 4, 40)])
def test_islands_equal_the_one_block_step(m3, spec, substeps, steps):
    _twins(m3, lambda: m3.World.scene(*spec), substeps, steps)


def test_a_kinematic_mover(m3):
    lib = abi.bind_create(m3.lib)
    lib.m3Body_SetType.argtypes = [abi.m3BodyId, C.c_int32]

    def between(w, step):
        if step == 5:
            body = abi.m3BodyId(9, w.id.index1 - 1, 0)
            lib.m3Body_SetType(body, 1)
            lib.m3Body_SetLinearVelocity(body, abi.m3Vec3(1.5, 0.0, 0.5))

    _twins(m3, lambda: m3.World.scene(SCENE_UNEVEN, 12, 300), 4, 30, between)
