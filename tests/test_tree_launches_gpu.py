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


@pytest.mark.parametrize("count", [16 * 148, 16 * 148 + 1])
def test_batches_about_the_early_line(m3, count):
    worlds = [m3.World.scene(SCENE_UNEVEN, 1 + i % 3, 6) for i in range(count)]
    alone = [m3.World.scene(SCENE_UNEVEN, 1 + i, 6) for i in range(3)]
    try:
        for steps in (3, 18):
            m3.step_worlds(worlds, DT, 2, steps)
            expected = []
            for w in alone:
                w.step(DT, 2, steps)
                expected.append(m3.snapshot(w))
            for i in (0, 1, 2, count - 3, count - 2, count - 1):
                assert m3.snapshot(worlds[i]) == expected[i % 3]
    finally:
        for w in worlds + alone:
            w.destroy()
