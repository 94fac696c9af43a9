"""When the tree's replays are launched (needs a B200).

Replays start after every step while a launch table is free, in gathers of
steps once all are in flight, and before anything that reads the tree.  A
world stepped in one call, in single calls or flushed after every step ends
in the same snapshot (tree nodes included), on either side of the table
count and of the ring's length.
"""
import pytest

from conftest import cuda_available
from maul3d_b200.abi import SCENE_MIXED, SCENE_UNEVEN

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

DT = 1.0 / 60.0


@pytest.mark.parametrize("spec,count", [((SCENE_MIXED, 4, 1500), 1), ((SCENE_UNEVEN, 6, 90), 5)])
@pytest.mark.parametrize("steps", [1, 15, 17, 33, 50])
def test_one_call_single_calls_and_flushes_agree(m3, spec, count, steps):
    def build():
        return [m3.World.scene(spec[0], spec[1] + i, spec[2]) for i in range(count)]

    together, single, flushed = build(), build(), build()
    try:
        m3.step_worlds(together, DT, 2, steps)
        for _ in range(steps):
            m3.step_worlds(single, DT, 2, 1)
            m3.step_worlds(flushed, DT, 2, 1)
            m3.flush_trees(flushed)
        expected = [m3.snapshot(w) for w in flushed]
        assert [m3.snapshot(w) for w in together] == expected
        assert [m3.snapshot(w) for w in single] == expected
    finally:
        for w in together + single + flushed:
            w.destroy()
