"""The workloads this library's step time is judged by, at the sizes it is used at.

A program steps a world, reads the states back, asks scene queries of it, differentiates through it
or calls the sort on its own; every case here is one such program's inner loop through the package's
entry points. The scenes are the generators of dynamis_b200.scenes at the sizes the benchmark, the
tests and the configurations use, and at sizes between them.

A simulated case starts every pass from one snapshot (as a planner or a trainer replays a rollout),
takes `steps` steps and reads every body state into pinned host memory, so each pass does the same
work. A resting world is at a fixed point, so it is stepped on without going back.

Single steps are reproducible bit for bit (fixed-point solver sums, contacts in pair order), so
states, query hits and sorted keys are compared exactly; only the gradients, whose shared rows are
summed with floating atomics in no fixed order, carry a tolerance.
"""
import ctypes
import math

import numpy as np
import torch

from dynamis_b200 import World, records as R, scenes
from dynamis_b200._native import check, lib
from dynamis_b200.autograd import rollout

# Bodies' contacts once the scene has formed (counted on the scenes below), for the traffic a step
# cannot do without.
CONTACTS_PER_BODY = {"heap": 2.0, "boxes": 2.5, "pile": 1.7, "chains": 0.2, "worlds": 2.2, "field": 1.0, "towers": 2.1}
STATE, DESC, COLLIDER, CONTACT, JOINT = 144, 128, 112, 352, 400


def listed():
    return [
        # one interactive object heap with every shape kind, pushed by one command a step: launches only
        {"name": "heap_64", "kind": "heap", "bodies": 64, "setup": 30, "steps": 16, "commands": 1},
        # the falling-boxes configuration, landed: a small world stepped in real time
        {"name": "boxes_1000", "kind": "boxes", "bodies": 1000, "setup": 60, "steps": 16},
        # a mid-sized pile with the options a game turns on: continuous collision on some bodies, the row-mass guard
        {"name": "pile_4913_ccd_guard", "kind": "pile", "side": 17, "setup": 90, "steps": 8, "ccd_every": 16, "guard": True},
        # the benchmark's mixed pile at an ordinary size and at its full one
        {"name": "pile_32768", "kind": "pile", "side": 32, "setup": 120, "steps": 8},
        {"name": "pile_262144", "kind": "pile", "side": 64, "setup": 120, "steps": 4},
        # the joint configuration: hanging chains of 32 boxes
        {"name": "chains_131072", "kind": "chains", "chains_x": 64, "chains_z": 64, "setup": 60, "steps": 4},
        # many small worlds in one launch, one command per world and step, as a learner drives them
        {"name": "worlds_1024", "kind": "worlds", "worlds": 1024, "setup": 30, "steps": 2, "commands": 1024},
        # a large world that has come to rest and is stepped every frame all the same
        {"name": "field_262144", "kind": "field", "side": 512, "setup": 60, "steps": 16},
        # a batch of scene queries on a formed pile: rays from above, sphere overlaps inside
        {"name": "queries_16384", "kind": "queries", "side": 32, "setup": 120, "queries": 16384},
        # the differentiable configuration: a rollout and its reverse
        {"name": "towers_64", "kind": "towers", "worlds": 64, "setup": 120, "steps": 20},
        # the sort on its own: pairs of words with a payload
        {"name": "sort_1048576", "kind": "sort", "keys": 1 << 20, "digits": 3},
    ]


def _between(rng, low, high):
    """A whole number in [low, high], even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["heap", "boxes", "pile", "chains", "worlds", "field", "queries", "towers", "sort"])
    if kind == "heap":
        n = _between(rng, 16, 512)
        return {"kind": kind, "bodies": n, "setup": rng.randint(20, 40), "steps": 16, "commands": rng.randint(0, 4)}
    if kind == "boxes":
        return {"kind": kind, "bodies": _between(rng, 100, 20000), "setup": rng.randint(45, 75), "steps": 8}
    if kind == "pile":
        case = {"kind": kind, "side": _between(rng, 8, 44), "setup": rng.randint(90, 130), "steps": 4}
        if rng.random() < 0.3:
            case["guard"] = True
        if rng.random() < 0.3:
            case["ccd_every"] = rng.randint(8, 64)
        return case
    if kind == "chains":
        return {"kind": kind, "chains_x": _between(rng, 2, 48), "chains_z": _between(rng, 2, 48),
                "setup": rng.randint(40, 70), "steps": 4}
    if kind == "worlds":
        n = _between(rng, 16, 700)
        return {"kind": kind, "worlds": n, "setup": rng.randint(20, 40), "steps": 2, "commands": rng.choice([0, n])}
    if kind == "field":
        return {"kind": kind, "side": _between(rng, 24, 400), "setup": 60, "steps": 16}
    if kind == "queries":
        return {"kind": kind, "side": _between(rng, 8, 36), "setup": rng.randint(90, 120), "queries": _between(rng, 64, 12000)}
    if kind == "towers":
        return {"kind": kind, "worlds": _between(rng, 4, 48), "setup": rng.randint(90, 120), "steps": rng.randint(11, 20)}
    return {"kind": kind, "keys": _between(rng, 1000, 3000000), "digits": rng.randint(1, 4)}


# ---- preparing ----
def _yawed_field(side, seed):
    """scenes.resting_field with a small seeded yaw per box (no box touches another)."""
    scene = scenes.resting_field(side)
    rng = np.random.default_rng(seed)
    scene.bodies["orientation"][:-1] = scenes.yaw_quaternions(rng.uniform(-0.05, 0.05, side * side))
    return scene


def _scene(case, seed):
    kind = case["kind"]
    if kind == "heap":
        # the heap's cube grows with its count, so the bodies overlap no deeper in a large one
        return scenes.random_mix(case["bodies"], seed=seed, extent=4.0 * (case["bodies"] / 64.0) ** (1.0 / 3.0))
    if kind == "boxes":
        return scenes.box_lattice(case["bodies"], seed)
    if kind in ("pile", "queries"):
        return scenes.mixed_pile(case["side"], seed=seed)
    if kind == "chains":
        return scenes.hanging_chains(case["chains_x"], case["chains_z"], 32, seed=seed)
    if kind == "worlds":
        # body counts log-uniform in [16, 2048] as scenes.batched_worlds draws them, the same ones for every seed
        counts = np.exp(np.random.default_rng(case["worlds"]).uniform(np.log(16), np.log(2048), case["worlds"])).astype(np.int64)
        return scenes.batch([scenes.box_lattice(int(n), seed * 100003 + w) for w, n in enumerate(counts)])
    if kind == "field":
        return _yawed_field(case["side"], seed)
    return scenes.differentiable_towers(case["worlds"], seed=seed)


def _dt(case):
    return 1.0 / 120.0 if case["kind"] in ("chains", "towers") else 1.0 / 60.0


class _Stepped:
    """A formed world, its snapshot, the pinned buffer its states are read into and its commands."""


def _form(case, seed):
    s = _Stepped()
    s.case, s.dt = case, _dt(case)
    scene = _scene(case, seed)
    options = {"sleep_time": float("inf")} if case["kind"] == "towers" else {}
    # reserve the pair stream for the formed scene, so no widening falls into a pass
    s.world = World(capacity={"pairs": 48 * max(len(scene.colliders), 256)}, **options)
    s.ids = scene.build(s.world)
    if case.get("guard"):
        s.world.set_solver_guard(R.SOLVER_GUARD_ROW_MASS)
    if case.get("ccd_every"):
        for body in s.ids[:-1:case["ccd_every"]]:
            s.world.set_ccd(int(body))
    for _ in range(case["setup"]):
        s.world.step(s.dt)
    s.world.wait()
    rows = s.world.sizes()["bodies"]
    s.pinned = torch.empty(rows * R.BODY_STATE.itemsize, dtype=torch.uint8).pin_memory()
    s.states = s.pinned.numpy().view(R.BODY_STATE)
    s.edits = None
    if case.get("commands"):
        rng = np.random.default_rng(seed + 1)
        count = case["commands"]
        if scene.worlds is not None:  # one body of each sub-world
            first = np.concatenate([[0], np.nonzero(np.diff(scene.worlds))[0] + 1])
            s.targets = s.ids[first[:count]]
        else:
            s.targets = s.ids[rng.choice(case["bodies"], min(count, case["bodies"]), replace=False)]
        s.edits = np.zeros(len(s.targets), R.BODY_EDIT)
        s.edits["kind"] = R.EDIT_IMPULSE
        s.edits["state"]["velocity"] = rng.normal(0.0, 50.0, (len(s.targets), 3)).astype(np.float32)
    return s


def _query_batch(world, count, seed):
    rng = np.random.default_rng(seed + 2)
    at = world.read_states()["position"][:-1]
    low, high = np.percentile(at, 1.0, axis=0), np.percentile(at, 99.0, axis=0)
    q = np.concatenate([R.ray_query((0, 1, 0), (0, -1, 0), 1.0, R.query_filter(max_hits=4)),
                        R.sphere_query((0, 0, 0), 0.75, R.query_filter(max_hits=8))])
    batch = q[np.arange(count) % 2]
    origins = rng.uniform(low, high, (count, 3)).astype(np.float32)
    rays = batch["kind"] == R.QUERY_RAY
    origins[rays, 1] = high[1] + 5.0
    batch["origin"] = origins
    batch["extent"][rays] = float(high[1] - low[1] + 10.0)
    return batch


def _keys(case, seed):
    """Major word, minor word and payload of every key."""
    generator = torch.Generator(device="cuda").manual_seed(seed)
    span = 1 << min(31, 8 * case["digits"])
    return torch.randint(0, span, (3, case["keys"]), dtype=torch.int32, device="cuda", generator=generator)


def prepare(case, seed):
    if case["kind"] == "sort":
        s = _Stepped()
        s.case, n = case, case["keys"]
        s.keys = _keys(case, seed)
        s.out = torch.empty_like(s.keys)
        s.stream = torch.cuda.Stream()
        s.world = World(capacity={"pairs": max(n, 1024)})
        s.world.set_stream(s.stream.cuda_stream)
        torch.cuda.synchronize()
        return s
    s = _form(case, seed)
    if case["kind"] == "queries":
        s.batch = _query_batch(s.world, case["queries"], seed)
        return s
    if case["kind"] == "towers":
        exported = s.world.export_scene()
        start = s.world.read_states()
        inverse = exported["descs"]["inverse_mass"]
        mass = np.where(inverse > 0, 1.0 / np.where(inverse > 0, inverse, 1.0), 0.0)
        spheres = np.sort(exported["owners"][exported["colliders"]["kind"] == R.SHAPE_SPHERE]).astype(np.int64)
        velocity = start["velocity"].copy()
        velocity[spheres] = scenes.sphere_launches(None, start, spheres, seed)
        s.parameters = [torch.tensor(x.astype(np.float32), requires_grad=True)
                        for x in (mass, exported["colliders"]["friction"], velocity)]
        rng = np.random.default_rng(seed + 3)
        s.target = torch.from_numpy((start["position"] + rng.normal(0.0, 0.05, start["position"].shape)).astype(np.float32))
    if case["kind"] != "field":
        s.snapshot = s.world.snapshot()
    return s


# ---- one pass ----
def _read(s):
    check(lib.dyn_download_states(s.world._h, s.pinned.data_ptr(), len(s.states)), s.world._h)
    return {name: s.states[name] for name in ("position", "orientation", "velocity", "angular_velocity", "sleep_timer",
                                              "sleeping", "body_id")}


def run(s):
    kind = s.case["kind"]
    if kind == "sort":
        digits = s.case["digits"]
        with torch.cuda.stream(s.stream):
            s.out.copy_(s.keys)
        major, minor, payload = (ctypes.c_void_p(s.out[i].data_ptr()) for i in range(3))
        check(lib.dyn_radix_sort(s.world._h, major, minor, payload, s.out.shape[1], digits, digits), s.world._h)
        return s.out
    if kind == "queries":
        queries, hits = s.world.query(s.batch)
        # query i's hits are hits[hit_base : hit_base + count]; the slots after them are not written
        slot = np.arange(len(hits)) - np.repeat(queries["hit_base"], queries["max_hits"])
        hits[slot >= np.repeat(queries["count"], queries["max_hits"])] = 0
        return {"count": queries["count"], "overflow": queries["overflow"],
                **{name: hits[name] for name in ("body_id", "distance", "point", "normal")}}
    if kind == "towers":
        s.world.restore(s.snapshot)
        for p in s.parameters:
            p.grad = None
        final = rollout(s.world, *s.parameters, s.case["steps"], s.dt)
        final.backward(2.0 * (final.detach() - s.target))
        return [final.detach()] + [p.grad for p in s.parameters]
    if kind != "field":
        s.world.restore(s.snapshot)
    for _ in range(s.case["steps"]):
        if s.edits is not None:
            s.world.edit_bodies(s.targets, s.edits)
        s.world.step(s.dt)
    return _read(s)


# ---- what a pass needs, and how close it comes ----
def _bodies(case):
    kind = case["kind"]
    if kind in ("heap", "boxes"):
        return case["bodies"]
    if kind in ("pile", "queries"):
        return case["side"] ** 3
    if kind == "chains":
        return case["chains_x"] * case["chains_z"] * 33
    if kind == "worlds":
        return int(case["worlds"] * (2048 - 16) / math.log(2048 / 16))
    if kind == "field":
        return case["side"] ** 2
    return case["worlds"] * 130


def work(case):
    kind = case["kind"]
    if kind == "sort":
        return {"bytes": 2 * 12.0 * case["keys"], "flops": 0}
    bodies = _bodies(case)
    if kind == "queries":
        return {"bytes": bodies * (STATE + COLLIDER) + case["queries"] * (2 * 144.0 + 48.0), "flops": 0}
    # a step: states read and written, descriptors and colliders read, last step's contacts read and this step's written
    step = bodies * (2 * STATE + DESC + COLLIDER + 2 * CONTACT * CONTACTS_PER_BODY[kind])
    if kind == "field":
        step = bodies * STATE  # nothing moves
    if kind == "chains":
        step += case["chains_x"] * case["chains_z"] * 32 * JOINT
    if kind == "towers":
        step *= 2  # the reverse reads what the step did
    return {"bytes": case["steps"] * step + bodies * STATE, "flops": 0}


def tolerance(case):
    if case["kind"] == "towers":
        # two runs of the same pass differ by 1.7e-7 (2-norm) and 1.2e-6 (largest) through the order of the
        # atomics alone; a sum over a body's contacts in another shape moves a few more last bits per step
        return {"rel": 1e-5, "max": 4e-4}
    return "exact"


def exact(case, seed):
    """The sort by numpy. A simulated step has no 64-bit value to be compared with: its solver sums are
    fixed-point words and its contact set is a decision of the 32-bit narrowphase."""
    if case["kind"] != "sort":
        return None
    keys = _keys(case, seed).cpu().numpy()
    mask = (1 << (8 * case["digits"])) - 1
    order = np.lexsort((keys[1] & mask, keys[0] & mask))
    return keys[:, order]
