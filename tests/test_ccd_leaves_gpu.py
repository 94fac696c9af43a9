"""The continuous phase against static bodies that were moved between steps
(needs a B200).

A fast body is swept against the static shapes whose tree leaves touch its
swept box (solver.c:3081-3274), the leaves as the step's own broadphase
left them (broad_phase.c:516-538): a static box teleported into a ball's
way must stop it in the very next step, in a world stepped alone, in a
batch whose replays start after every step, in one whose replays gather,
and in a served world, which keeps no tree.
"""
import ctypes as C

import pytest

from conftest import cuda_available
from maul3d_b200 import abi

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

DT = 1.0 / 60.0
# The ball moves 2 m a step from x = -5; the box's near face is at -4.2.
NEAR, RADIUS = -4.2, 0.2


def _world(m3):
    """A ball at 120 m/s (body 2) and a static box (body 1) far above."""
    lib = abi.bind_create(m3.lib)
    lib.m3Body_SetTransform.argtypes = [abi.m3BodyId, abi.m3Pos3, abi.m3Quat]
    lib.m3Body_SetTransform.restype = None
    wd = lib.m3DefaultWorldDef()
    wd.bodyCapacity = wd.shapeCapacity = 4
    wid = lib.m3CreateWorld(C.byref(wd))
    sd = lib.m3DefaultShapeDef()
    bd = lib.m3DefaultBodyDef()
    bd.position = abi.m3Pos3(0.0, 50.0, 0.0)
    box = lib.m3CreateBody(wid, C.byref(bd))
    lib.m3CreateBoxShape(box, C.byref(sd), abi.m3Vec3(0.5, 0.5, 0.5))
    bd = lib.m3DefaultBodyDef()
    bd.type = 2
    bd.position = abi.m3Pos3(-5.0, 5.0, 0.0)
    bd.linearVelocity = abi.m3Vec3(120.0, 0.0, 0.0)
    ball = lib.m3CreateBody(wid, C.byref(bd))
    lib.m3CreateSphereShape(ball, C.byref(sd),
                            C.byref(abi.m3Sphere(abi.m3Vec3(0.0, 0.0, 0.0), RADIUS)))
    return m3.World(wid), box


def _teleport(m3, box):
    m3.lib.m3Body_SetTransform(box, abi.m3Pos3(NEAR + 0.5, 5.0, 0.0),
                               abi.m3Quat(0.0, 0.0, 0.0, 1.0))


def _stopped(world):
    x = float(world.state().transforms["p"][1][0])
    assert -5.0 < x <= NEAR - RADIUS + 0.01, x


@pytest.mark.parametrize("early", [True, False])
def test_a_teleported_box_stops_the_ball_in_every_batch(m3, early):
    import torch
    # Replays start after every step up to 16 worlds an SM.
    count = 3 if early else 16 * torch.cuda.get_device_properties(0).multi_processor_count + 1
    alone, box = _world(m3)
    built = [_world(m3) for _ in range(count)]
    worlds = [w for w, _ in built]
    try:
        for b in [box] + [b for _, b in built]:
            _teleport(m3, b)
        alone.step(DT, 4, 1)
        m3.step_worlds(worlds, DT, 4, 1)
        expected = alone.hash()
        _stopped(alone)
        for w in worlds[:3] + worlds[-3:]:
            _stopped(w)
        assert [int(h) for h in m3.hash_worlds(worlds)] == [expected] * count
    finally:
        for w in worlds + [alone]:
            w.destroy()


def test_a_teleported_box_stops_the_ball_in_a_served_world(m3):
    world, box = _world(m3)
    _teleport(m3, box)
    container = abi.encode_container(m3.lib, m3.snapshot(world), abi.journal_step(DT, 4))
    server = m3.Server(device_budget=1 << 30, max_active=4)
    try:
        ticket = server.submit(container)
        served, status = server.run()[ticket]
        world.step(DT, 4, 1)
        _stopped(world)
        assert (served, status) == (world.hash(), 0)
    finally:
        server.close()
        world.destroy()
