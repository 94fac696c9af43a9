"""Kinematic targets on the wide path (needs a B200).

A step prepares its contact rows, with the closing speeds that restitution
uses, before the servo turns a kinematic body's target into velocities
(solver.c:3912-3983).  A platform carried against bouncing balls must give
the same world, every step, in one block and over the whole grid.
"""
import ctypes as C

import pytest

from conftest import cuda_available
from maul3d_b200 import abi

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

DT = 1.0 / 60.0


def _world(m3, restitution):
    lib = abi.bind_create(m3.lib)
    lib.m3Body_SetTargetTransform.argtypes = [abi.m3BodyId, abi.m3Pos3, abi.m3Quat]
    lib.m3Body_SetTargetTransform.restype = None
    wd = lib.m3DefaultWorldDef()
    wid = lib.m3CreateWorld(C.byref(wd))
    sd = lib.m3DefaultShapeDef()
    sd.restitution = restitution
    bd = lib.m3DefaultBodyDef()
    bd.type = 1
    platform = lib.m3CreateBody(wid, C.byref(bd))
    lib.m3CreateBoxShape(platform, C.byref(sd), abi.m3Vec3(3.0, 0.5, 3.0))
    for k in range(9):
        bd = lib.m3DefaultBodyDef()
        bd.type = 2
        bd.position = abi.m3Pos3(-2.0 + 2.0 * (k % 3), 1.0 + 0.1 * k, -2.0 + 2.0 * (k // 3))
        ball = lib.m3CreateBody(wid, C.byref(bd))
        lib.m3CreateSphereShape(ball, C.byref(sd),
                                C.byref(abi.m3Sphere(abi.m3Vec3(0.0, 0.0, 0.0), 0.5)))
    return m3.World(wid), platform


@pytest.mark.parametrize("restitution", [0.0, 0.7])
def test_a_carried_platform_is_the_same_on_both_paths(m3, restitution):
    def run(threshold):
        previous = m3.set_wide_min_shapes(threshold)
        world, platform = _world(m3, restitution)
        try:
            hashes = []
            for step in range(30):
                height = 0.15 * (step + 1) if step < 20 else 3.0 - 0.2 * (step - 19)
                m3.lib.m3Body_SetTargetTransform(platform, abi.m3Pos3(0.0, height, 0.0),
                                                 abi.m3Quat(0.0, 0.0, 0.0, 1.0))
                world.step(DT, 4, 1)
                hashes.append(world.hash())
            rise = float(world.state().transforms["p"][1][1])
            return hashes, rise
        finally:
            m3.set_wide_min_shapes(previous)
            world.destroy()

    block, rise = run(1 << 30)
    grid, _ = run(1)
    assert rise > 2.0  # the platform met the ball
    assert grid == block
