"""The work that programs using this library have it do, as timed cases.

Three kinds of program stand behind the cases:

  rollback  one world that a game simulates: it rewinds to a saved frame
            (a device snapshot slot), simulates some frames again with the
            players' inputs, hashes the result (peers compare hashes) and
            reads the whole state back to draw it;
  batch     many independent worlds of a training or search run: every
            world is rewound to its start state, the batch steps together
            for a rollout, every world's hash is read and the broadphase
            trees (snapshot state) are brought up to date;
  serve     a server answering replay containers (snapshot + journal of
            frames with impulses): all requests are submitted at once and
            the answer to each is its final world hash.

A pass always starts from the same saved state, so every pass does the
same work.  `exact` has no values: the step is a long chain of discrete
decisions (contact features, colours, breakage) whose result is defined
bit by bit.  A world's hash covers its whole state, every body, joint and
contact manifold byte for byte, and is compared as a whole number.
"""
from __future__ import annotations

import math

import numpy as np

import maul3d_b200 as m3
from maul3d_b200 import abi

DT = 1.0 / 60.0

SCENES = {
    "pyramid": abi.SCENE_BOX_PYRAMID,
    "uneven": abi.SCENE_UNEVEN,
    "towers": abi.SCENE_TOWERS,
    "terrain": abi.SCENE_TERRAIN,
    "bounce": abi.SCENE_BOUNCE,
    "city": abi.SCENE_CITY,
    "rain": abi.SCENE_RAIN,
    "mixed": abi.SCENE_MIXED,
}
# Seed of the body counts of a batch or of served requests (the counts are
# the same for every seed of a case; the worlds' contents differ).
SIZE_SEED = 20261203


def listed():
    return [
        # The smallest call: one frame of one small world (a few bodies
        # and three hinged chains), where launches and latency count.
        dict(name="rollback_uneven_32x1", kind="rollback", scene="uneven", size=32, substeps=4,
             warm=20, frames=1, inputs=2),
        # A wall of 210 boxes, eight frames re-simulated with inputs.
        dict(name="rollback_pyramid_210x8", kind="rollback", scene="pyramid", size=20, substeps=4,
             warm=30, frames=8, inputs=4),
        # A level of everyday size: stacks, spheres and chains.
        dict(name="rollback_uneven_485x8", kind="rollback", scene="uneven", size=485, substeps=4,
             warm=20, frames=8, inputs=4),
        # A large level of boxes, spheres and 16-point hulls, an odd size
        # just under the threshold where one world takes the whole GPU.
        dict(name="rollback_mixed_3001x4", kind="rollback", scene="mixed", size=3001, substeps=4,
             warm=20, frames=4, inputs=4),
        # 10,000 spheres, capsules and hulls falling on a heightfield: one
        # world over the whole GPU.
        dict(name="rollback_rain_10000x2", kind="rollback", scene="rain", size=10000, substeps=4,
             warm=24, frames=2, inputs=4),
        # 7,001 spheres, capsules and boxes piling up on rough ground: the
        # same path with contacts everywhere.
        dict(name="rollback_terrain_7001x4", kind="rollback", scene="terrain", size=7001,
             substeps=4, warm=20, frames=4, inputs=4),
        # 100 towers welded by 46,000 breakable joints under fire, eight
        # substeps a frame: one jointed world over the whole GPU.
        dict(name="rollback_city_100x2", kind="rollback", scene="city", size=100, substeps=8,
             warm=8, frames=2, inputs=4),
        # A small training batch.
        dict(name="batch_uneven_64x8", kind="batch", scene="uneven", worlds=64, lo=32, hi=2048,
             substeps=4, warm=20, frames=8),
        # The batched workload of uneven worlds.
        dict(name="batch_uneven_2048x8", kind="batch", scene="uneven", worlds=2048, lo=32, hi=2048,
             substeps=4, warm=20, frames=8),
        # Heightfield worlds.
        dict(name="batch_terrain_256x8", kind="batch", scene="terrain", worlds=256, lo=32, hi=512,
             substeps=4, warm=20, frames=8),
        # A thousand and one small worlds (restitution), long rollout.
        dict(name="batch_bounce_1001x16", kind="batch", scene="bounce", worlds=1001, lo=12, hi=96,
             substeps=2, warm=20, frames=16),
        # Served requests of 200 to 5000 bodies, 4 to 16 frames each.
        dict(name="serve_mixed_32", kind="serve", scene="mixed", requests=32, lo=200, hi=5000,
             substeps=4, warm=5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rollback", "rollback", "rollback", "batch", "batch", "serve"])
    if kind == "rollback":
        scene = rng.choice(["pyramid", "uneven", "uneven", "terrain", "bounce", "towers", "mixed",
                            "rain", "city"])
        lo, hi = {"pyramid": (4, 40), "uneven": (32, 3000), "terrain": (30, 7000),
                  "bounce": (16, 1500), "towers": (2, 60), "mixed": (50, 6000),
                  "rain": (500, 9000), "city": (1, 90)}[scene]
        size = _log_int(rng, lo, hi)
        large = scene in ("rain", "city") or size > 2500
        return dict(kind=kind, scene=scene, size=size, substeps=rng.choice([1, 2, 4, 4, 8]),
                    warm=rng.randint(4, 16) if large else rng.randint(4, 40),
                    frames=rng.randint(1, 2) if large else rng.randint(1, 12),
                    inputs=rng.randint(1, 8))
    if kind == "batch":
        scene = rng.choice(["uneven", "uneven", "terrain", "bounce", "mixed", "towers"])
        lo, hi, most = {"uneven": (32, 2048, 700), "terrain": (32, 512, 400),
                        "bounce": (12, 200, 1400), "mixed": (50, 600, 400),
                        "towers": (1, 12, 500)}[scene]
        a = _log_int(rng, lo, hi)
        b = _log_int(rng, lo, hi)
        return dict(kind=kind, scene=scene, worlds=_log_int(rng, 8, most), lo=min(a, b),
                    hi=max(a, b) + 1, substeps=rng.choice([2, 4, 4, 8]), warm=rng.randint(4, 30),
                    frames=rng.randint(1, 8))
    a = _log_int(rng, 100, 4000)
    b = _log_int(rng, 100, 4000)
    return dict(kind=kind, scene="mixed", requests=_log_int(rng, 2, 28), lo=min(a, b),
                hi=max(a, b) + 1, substeps=4, warm=rng.randint(2, 8))


def _sizes(case, count):
    return [int(m3.lib.m3s_uneven_size(SIZE_SEED, i, case["lo"], case["hi"]))
            for i in range(count)]


def _world(scene, seed, size):
    return m3.World.scene(SCENES[scene], seed, size)


class _Worlds:
    """Worlds that leave the device with the state that holds them."""

    def __init__(self, worlds):
        self.batch = m3.WorldBatch(worlds)

    def __del__(self):
        for w in self.batch.worlds:
            w.destroy()


class _Server:
    def __init__(self):
        self.server = m3.Server(device_budget=16 << 30, max_active=1024)

    def __del__(self):
        self.server.close()


def _inputs(rng, count, worlds, bodies):
    """`count` impulses of 1 to 20 N s on random bodies of the worlds, for
    one frame."""
    out = []
    for _ in range(count):
        d = rng.normal(size=3)
        d *= rng.uniform(1.0, 20.0) / np.linalg.norm(d)
        wi = int(rng.integers(len(worlds)))
        body = abi.m3BodyId(int(rng.integers(2, bodies[wi] + 1)), worlds[wi].id.index1 - 1, 0)
        out.append((wi, abi.OP_APPLY_LINEAR_IMPULSE, body, tuple(float(x) for x in d)))
    return out


def _containers(case, rng, seed):
    out = []
    for i, size in enumerate(_sizes(case, case["requests"])):
        w = _world(case["scene"], seed * 4099 + i, size)
        w.step(DT, case["substeps"], case["warm"])
        bodies = w.body_count()
        journal = b""
        for _ in range(4 + (5 * i) % 13):
            for _ in range(int(rng.integers(1, 9))):
                d = rng.normal(size=3)
                d *= rng.uniform(1.0, 50.0) / np.linalg.norm(d)
                journal += abi.journal_body_command(abi.OP_APPLY_LINEAR_IMPULSE,
                                                    int(rng.integers(2, bodies + 1)), 0,
                                                    [float(x) for x in d])
            journal += abi.journal_step(DT, case["substeps"])
        out.append(abi.encode_container(m3.lib, m3.snapshot(w), journal))
        w.destroy()
    return out


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "serve":
        return dict(case=case, containers=_containers(case, rng, seed), server=_Server())
    if case["kind"] == "rollback":
        worlds = [_world(case["scene"], seed * 4099 + 17, case["size"])]
    else:
        worlds = [_world(case["scene"], seed * 4099 + i, n)
                  for i, n in enumerate(_sizes(case, case["worlds"]))]
    held = _Worlds(worlds)
    batch = held.batch
    bodies = [w.body_count() for w in worlds]
    # A first frame with inputs from the seed, then the worlds settle in.
    m3.step_worlds_commands(batch, _inputs(rng, 4 * len(worlds), worlds, bodies), DT,
                            case["substeps"])
    m3.step_worlds(batch, DT, case["substeps"], case["warm"])
    m3.flush_trees(batch)
    for w in worlds:
        w.reserve_slots(1)
        w.save_slot(0)
    frames = []
    if case["kind"] == "rollback":
        frames = [_inputs(rng, case["inputs"], worlds, bodies) for _ in range(case["frames"])]
    return dict(case=case, held=held, frames=frames)


def run(state):
    case = state["case"]
    if case["kind"] == "serve":
        server = state["server"].server
        tickets = [server.submit(c) for c in state["containers"]]
        done = server.run()
        return {"hash": np.array([done[t][0] for t in tickets], np.uint64),
                "status": np.array([done[t][1] for t in tickets], np.int32)}
    batch = state["held"].batch
    for w in batch:
        w.restore_slot(0)
    if case["kind"] == "batch":
        m3.step_worlds(batch, DT, case["substeps"], case["frames"])
        hashes = m3.hash_worlds(batch).copy()
        m3.flush_trees(batch)
        return {"hash": hashes}
    for inputs in state["frames"]:
        m3.step_worlds_commands(batch, inputs, DT, case["substeps"])
    world = batch.worlds[0]
    value = world.hash()
    s = world.state()
    return {"hash": np.array([value], np.uint64), "position": s.transforms["p"], "rotation": s.transforms["q"],
            "linear": s.lin, "angular": s.ang, "awake": s.awake, "sleep_time": s.sleep}


def _counts(case):
    """Dynamic bodies, joints, frames of a case (all worlds together),
    frames weighted by bodies for served requests."""
    if case["kind"] == "rollback":
        scene, size = case["scene"], case["size"]
        bodies = {"pyramid": size * (size + 1) // 2, "towers": 17 * size,
                  "city": 204 * size}.get(scene, size)
        joints = {"towers": 28 * size, "city": 460 * size, "uneven": 24}.get(scene, 0)
        return bodies, joints, case["frames"]
    if case["kind"] == "batch":
        size = sum(_sizes(case, case["worlds"]))
        if case["scene"] == "towers":
            return 17 * size, 28 * size, case["frames"]
        return size, 24 * case["worlds"] if case["scene"] == "uneven" else 0, case["frames"]
    sizes = _sizes(case, case["requests"])
    frames = sum(n * (4 + (5 * i) % 13) for i, n in enumerate(sizes)) / sum(sizes)
    return sum(sizes), 0, frames


def work(case):
    """The state in and out once (about 400 bytes a body with its shape,
    300 a joint, two contact pairs of 196 bytes a body), and the
    arithmetic of a step: about 3,000 operations of broad- and narrowphase
    a body, and per substep 200 a body, three passes of 400 a contact pair
    and of 400 a joint."""
    bodies, joints, frames = _counts(case)
    pairs = 2 * bodies
    moved = 400 * bodies + 300 * joints + 196 * pairs
    per_substep = 200 * bodies + 1200 * pairs + 1200 * joints
    return {"bytes": 2 * moved,
            "flops": frames * (3000 * bodies + case["substeps"] * per_substep)}


def exact(case, seed):
    return None
