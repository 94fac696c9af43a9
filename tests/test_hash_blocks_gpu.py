"""World hashes over many blocks against the host's fold (needs a B200).

The host folds the stream byte by byte (m3_hash.h; snapshot.c:932-1345 of
the reference).  Worlds on both sides of the record count from which a
world is hashed over many blocks, one of exactly whole and one of partial
8 KB tiles' worth of records, one with joints and thousands of pairs, one
with every optional field of a body, and batches of as many large worlds
as the passes take at once, one more, and with small worlds among them.
"""
import pytest

from conftest import cuda_available
from maul3d_b200 import abi
from maul3d_b200.abi import (SCENE_BOUNCE, SCENE_CITY, SCENE_FREEFALL, SCENE_MIXED, SCENE_TERRAIN,
                             SCENE_UNEVEN)

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

DT = 1.0 / 60.0


def _check(m3, worlds):
    got = [int(h) for h in m3.hash_worlds(worlds)]
    for w, h in zip(worlds, got):
        w.state()  # the host image is current again: its hash folds on the host
        assert w.hash() == h


@pytest.mark.parametrize("spec", [
    (SCENE_FREEFALL, 0, 126), (SCENE_FREEFALL, 0, 127), (SCENE_FREEFALL, 0, 128),
    (SCENE_FREEFALL, 0, 129), (SCENE_UNEVEN, 3, 115), (SCENE_UNEVEN, 3, 1023),
    (SCENE_TERRAIN, 4, 900), (SCENE_MIXED, 5, 2047), (SCENE_CITY, 6, 7)])
def test_one_world(m3, spec):
    w = m3.World.scene(*spec)
    for steps in (1, 3):
        w.step(DT, 4, steps)
        _check(m3, [w])
    w.destroy()


def test_optional_body_fields(m3):
    w = m3.World.scene(SCENE_UNEVEN, 8, 400)
    lib = abi.bind_create(m3.lib)
    w0 = w.id.index1 - 1
    for k in range(2, 300):
        b = abi.m3BodyId(k, w0, 0)
        lib.m3Body_ApplyForce(b, abi.m3Vec3(0.5 * k, 1.0, -2.0))
    m3.upload_worlds([w])
    _check(m3, [w])
    w.step(DT, 2, 2)
    _check(m3, [w])
    w.destroy()


@pytest.mark.parametrize("large,small", [(63, 5), (64, 0), (65, 3)])
def test_batches(m3, large, small):
    worlds = [m3.World.scene(SCENE_UNEVEN, 20 + k, 130 + k) for k in range(large)]
    worlds += [m3.World.scene(SCENE_BOUNCE, 20 + k, 5 + k) for k in range(small)]
    m3.step_worlds(worlds, DT, 4, 2)
    _check(m3, worlds)
    for w in worlds:
        w.destroy()
