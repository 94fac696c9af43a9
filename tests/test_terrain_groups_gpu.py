"""Heightfield pairs by groups of lanes against one thread a pair (needs a
B200).

The batched step gives a heightfield pair with a capsule or a hull a group
of eight lanes, or a warp when more than 32 triangles are near; the
allocation-free step gives every pair one thread.  Both step twin worlds:
bodies smaller than a cell, long capsules and wide hulls over dozens of
triangles (the 64-candidate lists full), pair counts that leave a warp's
last groups empty, bodies over the grid's edge and off it.  Every step's
hash must be the same, alone and in a batch.
"""
import ctypes as C

import numpy as np
import pytest

from conftest import cuda_available
from maul3d_b200 import abi

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

DT = 1.0 / 60.0


def _world(lib, kind: str, count: int):
    rng = np.random.default_rng(100 + count)
    wd = lib.m3DefaultWorldDef()
    wd.bodyCapacity = wd.shapeCapacity = count + 1
    wid = lib.m3CreateWorld(C.byref(wd))
    sd = lib.m3DefaultShapeDef()
    n, cell = 41, 0.5
    heights = (0.25 * rng.random(n * n)).astype(np.float32)
    ground = lib.m3CreateBody(wid, C.byref(lib.m3DefaultBodyDef()))
    lib.m3CreateHeightFieldGridShape(ground, C.byref(sd),
                                     heights.ctypes.data_as(C.POINTER(C.c_float)), n, n, cell)
    for k in range(count):
        bd = lib.m3DefaultBodyDef()
        bd.type = 2
        wide = kind == "wide"
        x, z = rng.uniform(-1.0, 21.0, 2)
        y = (1.0 if wide else 0.6) + (3.0 if wide else 0.8) * k
        bd.position = abi.m3Pos3(float(x), float(y), float(z))
        bd.linearVelocity = abi.m3Vec3(0.0, -4.0 - 0.2 * k, 0.0)
        if not wide:
            bd.position = abi.m3Pos3(float(x), float(0.45 + 0.1 * rng.random()), float(z))
        body = lib.m3CreateBody(wid, C.byref(bd))
        size = float(rng.uniform(2.0, 5.0) if wide else rng.uniform(0.15, 0.4))
        if k % 3 == 0:
            cap = abi.m3Capsule(abi.m3Vec3(-size, 0.0, 0.0), abi.m3Vec3(size, 0.0, 0.1),
                                0.25 * min(size, 2.0))
            lib.m3CreateCapsuleShape(body, C.byref(sd), C.byref(cap))
        elif k % 3 == 1:
            lib.m3CreateBoxShape(body, C.byref(sd), abi.m3Vec3(size, 0.3, 0.8 * size))
        else:
            pts = (abi.m3Vec3 * 20)()
            for i, p in enumerate(rng.normal(size=(20, 3))):
                p *= size / np.linalg.norm(p)
                pts[i] = abi.m3Vec3(float(p[0]), float(0.4 * p[1]), float(p[2]))
            lib.m3CreateHullShape(body, C.byref(sd), pts, 20)
    return wid


@pytest.mark.parametrize("kind,count", [("small", 1), ("small", 2), ("small", 3), ("small", 7),
                                        ("small", 50), ("small", 203), ("wide", 1), ("wide", 2),
                                        ("wide", 3), ("wide", 9)])
def test_groups_equal_threads(m3, kind, count):
    lib = abi.bind_create(m3.lib)
    lib.m3gpu_step_world_noalloc.argtypes = [abi.m3WorldId, C.c_float, C.c_int32]
    thread, alone, batched = (m3.World(_world(lib, kind, count)) for _ in range(3))
    others = [m3.World(_world(lib, "small", 4 + k)) for k in range(5)]
    m3.reserve_worlds([thread])
    m3.upload_worlds([thread])
    contacts = 0
    for step in range(24):
        assert lib.m3gpu_step_world_noalloc(thread.id, DT, 4) == 0
        alone.step(DT, 4, 1)
        m3.step_worlds([batched] + others, DT, 4, 1)
        want = thread.hash()
        assert alone.hash() == want, f"alone, step {step + 1}"
        assert batched.hash() == want, f"batched, step {step + 1}"
        contacts = max(contacts, int(alone.state().manifolds["pointCount"].sum()))
    assert contacts > 0
    for w in (thread, alone, batched, *others):
        w.destroy()
