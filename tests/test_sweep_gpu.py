"""The broadphase's pair list against brute force (needs a B200).

Worlds of static and dynamic spheres: a sphere's fresh bounds are its
centre plus and minus (radius + margin) in double (broad_phase.c:22-135),
and the pair list after a step holds exactly the pairs whose bounds
overlap and that are not both static, in ascending order
(broad_phase.c:641-681).  Sizes around the powers of two the sort pads
to, around the wide path's 2048-element chunks, and piles: spheres wide
enough to overlap most of the world (the sweep's long positions, more of
them than the block's list holds) and so many overlapping static spheres
that the candidate list overflows.  Every world runs as one block and
over the whole grid.
"""
import ctypes as C

import numpy as np
import pytest

from conftest import cuda_available
from maul3d_b200 import abi

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]


def _spheres(kind: str, n: int):
    """Centres, radii and which are dynamic, on a seeded layout."""
    rng = np.random.default_rng(n)
    side = max(2.0, 2.2 * n ** (1.0 / 3.0))
    centre = rng.uniform(-side / 2, side / 2, (n, 3))
    radius = rng.uniform(0.3, 0.7, n).astype(np.float32)
    dynamic = rng.random(n) < 0.5
    if kind == "wide":
        # A few spheres reach across the world; all others are small.
        radius *= np.float32(0.4)
        big = rng.permutation(n)[:max(1, min(100, n // 8))]
        dynamic[:] = True
        dynamic[big] = False
        centre[big, 1] -= side * 4
        radius[big] = np.float32(4.2 * side)
        dynamic[rng.permutation(n)[:n - max(4, n // 16)]] = False
    elif kind == "pile":
        centre *= 0.02
        dynamic[:] = False
        dynamic[rng.permutation(n)[:5]] = True
    return centre, radius, dynamic


def _world(lib, centre, radius, dynamic):
    wd = lib.m3DefaultWorldDef()
    wd.bodyCapacity = wd.shapeCapacity = len(radius)
    wid = lib.m3CreateWorld(C.byref(wd))
    sd = lib.m3DefaultShapeDef()
    for c, r, d in zip(centre, radius, dynamic):
        bd = lib.m3DefaultBodyDef()
        bd.type = 2 if d else 0
        bd.position = abi.m3Pos3(*[float(x) for x in c])
        body = lib.m3CreateBody(wid, C.byref(bd))
        lib.m3CreateSphereShape(body, C.byref(sd), C.byref(abi.m3Sphere(abi.m3Vec3(0, 0, 0), r)))
    return wid


def _expected(centre, radius, dynamic):
    fat = (radius + np.float32(4.0) * np.float32(0.005)).astype(np.float64)[:, None]
    lo, hi = centre - fat, centre + fat
    keys = []
    for i in range(len(radius)):
        j = np.arange(i + 1, len(radius))
        hit = np.all((lo[i] <= hi[j]) & (lo[j] <= hi[i]), axis=1) & (dynamic[i] | dynamic[j])
        keys.append((np.uint64(i) << np.uint64(32)) | j[hit].astype(np.uint64))
    return np.concatenate(keys)


@pytest.mark.parametrize("kind,n", [
    ("spread", 1), ("spread", 2), ("spread", 3), ("spread", 255), ("spread", 256),
    ("spread", 257), ("spread", 2047), ("spread", 2048), ("spread", 2049), ("spread", 4096),
    ("spread", 4097), ("spread", 6200), ("wide", 40), ("wide", 700), ("wide", 2500),
    ("pile", 200), ("pile", 1100)])
def test_pairs_equal_brute_force(m3, kind, n):
    lib = abi.bind_create(m3.lib)
    centre, radius, dynamic = _spheres(kind, n)
    want = _expected(centre, radius, dynamic)
    assert 0 < len(want) <= 8 * n or n < 4
    previous = m3.set_wide_min_shapes(0)
    for threshold in (1 << 30, 1):
        m3.set_wide_min_shapes(threshold)
        try:
            w = m3.World(_world(lib, centre, radius, dynamic))
            w.step(1.0 / 60.0, 1, 1)
            assert np.array_equal(w.state().keys, want), f"wide threshold {threshold}"
            w.destroy()
        finally:
            m3.set_wide_min_shapes(previous)
