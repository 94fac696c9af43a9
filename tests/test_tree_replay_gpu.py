"""The device's replay of leaf moves into the broadphase tree (needs a
B200).

A world steps on the device; its twin stays on the host.  After every
step the leaves whose boxes the device changed are moved in the twin, in
ascending shape order, by the plain operations that build every tree at
creation (m3_tree.h; dynamic_tree.c:205-358 of the reference), and the
two trees must be equal byte for byte.  The sizes are the edges of the
replay: a tree of one leaf, of two (the root is a leaf's parent), of
three, one chunk of 32 moves and one more, and trees whose insertions
leave nodes out of balance.  A tree whose inner box is not the union of
its children's (a restored snapshot may hold one) is replayed without
stopping early.
"""
import ctypes as C
import struct

import numpy as np
import pytest

from conftest import cuda_available
from maul3d_b200 import abi
from maul3d_b200.abi import SCENE_FREEFALL, SCENE_RAIN, SCENE_UNEVEN

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

DT = 1.0 / 60.0
NODE = np.dtype([("box", "<f8", 6), ("parent", "<i4"), ("child1", "<i4"), ("child2", "<i4"),
                 ("shape", "<i4"), ("height", "<i4"), ("pad", "<i4")])


def _move(lib, world, shape, box) -> int:
    lib.m3gpu_tree_move.argtypes = [abi.m3WorldId, C.c_int32, C.c_void_p, C.c_void_p]
    lib.m3gpu_tree_move.restype = C.c_int32
    box = np.ascontiguousarray(box, np.float64)
    leaf = lib.m3gpu_tree_move(world.id, int(shape), box[:3].ctypes.data, box[3:].ctypes.data)
    assert leaf >= 0
    return leaf


def _layout(m3, spec, shape):
    """Offset of the tree's nodes in a snapshot of the scene and their
    count: a leaf is given a box found nowhere else."""
    w = m3.World.scene(*spec)
    box = [1234.5625, -77.125, 3.0625, 1235.5625, -76.125, 4.0625]
    leaf = _move(m3.lib, w, shape, box)
    snap = m3.snapshot(w)
    w.destroy()
    at = snap.find(struct.pack("<6d", *box))
    return at - NODE.itemsize * leaf, 2 * struct.unpack_from("<i", snap, 44)[0]


def _nodes(snap, layout):
    return np.frombuffer(snap, NODE, layout[1], layout[0])


def _replay(m3, device, twin, layout, steps):
    """Steps the device world and moves the twin's leaves the same way;
    both trees after every step."""
    for step in range(steps):
        device.step(DT, 4, 1)
        want = _nodes(m3.snapshot(twin), layout)
        got = _nodes(m3.snapshot(device), layout)
        box = {int(n["shape"]): n["box"] for n in got[got["height"] == 0]}
        for n in sorted(want[want["height"] == 0], key=lambda n: int(n["shape"])):
            shape = int(n["shape"])
            if box[shape].tobytes() != n["box"].tobytes():
                _move(m3.lib, twin, shape, box[shape])
        want = _nodes(m3.snapshot(twin), layout)
        assert got.tobytes() == want.tobytes(), f"step {step + 1}"


@pytest.mark.parametrize("spec,shape,steps", [
    ((SCENE_FREEFALL, 0, 1), 0, 6), ((SCENE_FREEFALL, 0, 2), 1, 6),
    ((SCENE_FREEFALL, 0, 3), 1, 6), ((SCENE_FREEFALL, 0, 32), 1, 6),
    ((SCENE_FREEFALL, 0, 33), 1, 6), ((SCENE_UNEVEN, 5, 150), 3, 30),
    ((SCENE_RAIN, 6, 700), 3, 20)])
def test_replayed_tree_equals_the_plain_operations(m3, spec, shape, steps):
    layout = _layout(m3, spec, shape)
    device, twin, whole = (m3.World.scene(*spec) for _ in range(3))
    _replay(m3, device, twin, layout, steps)
    # All steps in one call, replayed from the ring, give the same bytes.
    whole.step(DT, 4, steps)
    assert m3.snapshot(whole) == m3.snapshot(device)
    for w in (device, twin, whole):
        w.destroy()


def test_a_tree_with_a_loose_inner_box_is_walked_to_the_root(m3):
    abi.bind_snapshot(m3.lib)
    spec = (SCENE_RAIN, 6, 400)
    layout = _layout(m3, spec, 3)
    device, twin = (m3.World.scene(*spec) for _ in range(2))
    snap = bytearray(m3.snapshot(twin))
    nodes = np.frombuffer(snap, NODE, layout[1], layout[0])
    loose = int(np.argmax(nodes["height"] == 4))
    nodes["box"][loose, 0] -= 3.0
    data = (C.c_uint8 * len(snap)).from_buffer_copy(snap)
    for w in (device, twin):
        assert m3.lib.m3World_Restore(w.id, data, len(snap))
    _replay(m3, device, twin, layout, 8)
    for w in (device, twin):
        w.destroy()
