"""The broadphase where fewer shapes are swept than there are slots (needs
a B200).

Planes and dead slots (of a restored snapshot) take a slot but are not
swept, so slots and swept shapes can lie on different sides of the size up
to which a world's sort fits shared memory (4,096), of a power of two, or
leave holes in a 2,048-element chunk of the wide sort.  The pair list must
equal brute force (broad_phase.c:641-681; a plane pairs with every shape
the filter allows) in a call of two worlds (a block each), alone as one
block and alone over the whole grid, and the three must hash the same.
"""
import ctypes as C

import numpy as np
import pytest

from conftest import cuda_available
from maul3d_b200 import abi

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

DT = 1.0 / 60.0


def _layout(n: int, planes: int):
    """Per slot: whether it is a plane (spread over the slots), and the
    spheres' centres, radii and which are dynamic."""
    total = n + planes
    plane = np.zeros(total, bool)
    plane[(np.arange(planes) * total) // max(planes, 1) + total // (2 * max(planes, 1))] = True
    rng = np.random.default_rng(total)
    side = 2.2 * n ** (1.0 / 3.0)
    centre = rng.uniform(-side / 2, side / 2, (total, 3))
    radius = rng.uniform(0.3, 0.7, total).astype(np.float32)
    dynamic = (rng.random(total) < 0.3) & ~plane
    return plane, centre, radius, dynamic


def _world(m3, layout):
    plane, centre, radius, dynamic = layout
    lib = abi.bind_create(m3.lib)
    wd = lib.m3DefaultWorldDef()
    wd.bodyCapacity = wd.shapeCapacity = len(radius)
    wid = lib.m3CreateWorld(C.byref(wd))
    sd = lib.m3DefaultShapeDef()
    for p, c, r, d in zip(plane, centre, radius, dynamic):
        bd = lib.m3DefaultBodyDef()
        bd.type = 2 if d else 0
        bd.position = abi.m3Pos3(*[float(x) for x in c])
        body = lib.m3CreateBody(wid, C.byref(bd))
        if p:
            # Far below: a pair, never a contact.
            lib.m3CreatePlaneShape(body, C.byref(sd),
                                   C.byref(abi.m3Plane(abi.m3Vec3(0, 1, 0), -1000.0)))
        else:
            lib.m3CreateSphereShape(body, C.byref(sd),
                                    C.byref(abi.m3Sphere(abi.m3Vec3(0, 0, 0), r)))
    return m3.World(wid)


def _expected(layout, alive):
    plane, centre, radius, dynamic = layout
    fat = (radius + np.float32(4.0) * np.float32(0.005)).astype(np.float64)[:, None]
    lo, hi = centre - fat, centre + fat
    keys = []
    for i in np.flatnonzero(alive):
        j = np.arange(i + 1, len(radius))
        hit = np.all((lo[i] <= hi[j]) & (lo[j] <= hi[i]), axis=1) | plane[i] | plane[j]
        hit &= (dynamic[i] | dynamic[j]) & alive[j]
        keys.append((np.uint64(i) << np.uint64(32)) | j[hit].astype(np.uint64))
    return np.concatenate(keys)


def _kill(m3, snap, slots, dead):
    """The snapshot with shape slots `dead` not alive.  The liveness block
    lies before the shapes' free queue, the pair keys (eight a slot), the
    proxies and the tree's nodes (snapshot.c:161-678), whose place a leaf
    with a box found nowhere else gives."""
    probe = _world(m3, _layout(slots, 0))
    lib = m3.lib
    lib.m3gpu_tree_move.argtypes = [abi.m3WorldId, C.c_int32, C.c_void_p, C.c_void_p]
    lib.m3gpu_tree_move.restype = C.c_int32
    box = np.array([1234.5625, -77.125, 3.0625, 1235.5625, -76.125, 4.0625])
    leaf = lib.m3gpu_tree_move(probe.id, 3, box[:3].ctypes.data, box[3:].ctypes.data)
    nodes = m3.snapshot(probe).find(box.tobytes()) - 72 * leaf
    probe.destroy()
    alive = nodes - (4 + 64 + 4 + 1) * slots
    out = bytearray(snap)
    assert out[alive:alive + slots] == b"\x01" * slots
    for k in dead:
        out[alive + int(k)] = 0
    return bytes(out)


def _check(m3, build, want):
    previous = m3.set_wide_min_shapes(0)
    hashes = []
    try:
        for threshold, count in ((previous, 2), (1 << 30, 1), (1, 1)):
            m3.set_wide_min_shapes(threshold)
            worlds = [build() for _ in range(count)]
            m3.step_worlds(worlds, DT, 1, 1)
            for w in worlds:
                keys = w.state().keys
                assert np.array_equal(keys, want), f"threshold {threshold}, {count} worlds"
            m3.step_worlds(worlds, DT, 2, 4)
            hashes += [int(h) for h in m3.hash_worlds(worlds)]
            for w in worlds:
                w.destroy()
    finally:
        m3.set_wide_min_shapes(previous)
    assert hashes == [hashes[0]] * 4


@pytest.mark.parametrize("n,planes", [(256, 1), (2048, 1), (2040, 8), (4096, 1), (4090, 8),
                                      (4095, 1), (4097, 1)])
def test_planes_among_the_slots(m3, n, planes):
    layout = _layout(n, planes)
    want = _expected(layout, np.ones(n + planes, bool))
    assert 0 < len(want) <= 8 * (n + planes)
    _check(m3, lambda: _world(m3, layout), want)


@pytest.mark.parametrize("slots,living", [(300, 250), (2500, 2048), (5000, 3900), (5000, 4096),
                                          (5000, 4097), (9000, 3900)])
def test_dead_slots_of_a_restored_snapshot(m3, slots, living):
    layout = _layout(slots, 0)
    alive = np.zeros(slots, bool)
    alive[np.random.default_rng(living).permutation(slots)[:living]] = True
    source = _world(m3, layout)
    snap = _kill(m3, m3.snapshot(source), slots, np.flatnonzero(~alive))
    source.destroy()
    want = _expected(layout, alive)
    assert 0 < len(want) <= 8 * slots

    def build():
        w = _world(m3, layout)
        buf = (C.c_uint8 * len(snap)).from_buffer_copy(snap)
        assert m3.lib.m3World_Restore(w.id, buf, len(snap))
        return w

    _check(m3, build, want)
