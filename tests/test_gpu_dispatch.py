"""The batch-size dispatches and tile edges of the step's kernels, each against its reference.

* The GJK runs a pair on a lane group up to 8,192 pairs and on a lane above that: piles on both
  sides of the line are compared with the oracle, contact for contact.
* The coarse pair walk gives a thread one cell up to 8,192 colliders and a level slice above: fields
  just below and above the line give the oracle's pair list.
* The sorts' tiles hold 2,048 keys up to 303,104 and 4,096 above, and up to three grid runs share a
  sort's launches: key counts at the tile edges and on both sides of the line against numpy, and a
  half-resting world against the oracle.
* A query batch of up to two an SM goes to blocks, a larger one to warps, which hand on to blocks
  the queries that keep more than 512 candidates or, up to eight queries an SM, cover many cells.
* A restored world repeats its steps, its contact stream far from full.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from dynamis_b200 import World, records as R, scenes
from dynamis_b200._native import check, lib
from oracle.oracle import OracleWorld, oracle_from_world
from test_gpu_parity import compare_step
from test_gpu_query import compare as compare_queries

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def oracle_at(world):
    """The oracle over the device's current states, without archived contacts."""
    scene = world.export_scene()
    scene["states"] = world.read_states()
    return OracleWorld(scene, world.step_params(DT))


@pytest.mark.parametrize("side", [14, 26])
def test_gjk_batches_on_both_sides_of_the_group_line(side):
    # 2,744 bodies reach the GJK with about 1,500 pairs, 17,576 with about 11,000
    formed = World()
    scene = scenes.mixed_pile(side, seed=3)
    scene.build(formed)
    for _ in range(110):
        formed.step(DT)
    states = formed.read_states()
    formed.close()
    world = World()
    scene.build(world)
    world.upload_states(states)
    oracle = oracle_at(world)
    world.step(DT)
    oracle.step(DT)
    world.wait()
    assert (world.debug_paths()["gjk_pairs"] > 8192) == (side == 26)
    compare_step(world, oracle, 0)
    world.close()


@pytest.mark.parametrize("side", [90, 91])
def test_coarse_walk_on_both_sides_of_the_split(side):
    # 8,101 and 8,282 colliders; the plane makes every box a coarse link
    scene = scenes.resting_field(side)
    rng = np.random.default_rng(side)
    scene.bodies["position"][:-1] += rng.uniform(-0.3, 0.3, (side * side, 3)).astype(np.float32)
    scene.colliders["half_extents"][:-1] *= rng.uniform(0.4, 2.5, (side * side, 1)).astype(np.float32)
    world = World(capacity={"pairs": 1 << 20})
    scene.build(world)
    oracle = oracle_from_world(world, DT)
    world.step(DT)
    oracle.step(DT)
    world.wait()
    gpu, ref = world.debug_pairs(), oracle.pairs()
    assert np.array_equal(gpu[0], ref[0]) and np.array_equal(gpu[1], ref[1])
    world.close()


@pytest.mark.parametrize("n", [2047, 2048, 2049, 4095, 4096, 4097, 8191, 8192, 8193, 3 * 4096 + 1, 148 * 2048, 148 * 2048 + 1,
                               80 * 4096, 80 * 4096 + 1])
@pytest.mark.parametrize("words", [1, 2])
def test_sort_at_the_tile_edges(n, words):
    rng = np.random.default_rng(n + words)
    # few distinct keys, so that the order of equal ones shows
    keys = rng.integers(0, 700, (words, n), dtype=np.int64).astype(np.int32)
    world = World(capacity={"pairs": 1 << 19})
    tensors = [torch.from_numpy(k.copy()).cuda() for k in keys]
    payload = torch.arange(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    minor = tensors[1].data_ptr() if words == 2 else None
    check(lib.dyn_radix_sort(world._h, tensors[0].data_ptr(), minor, payload.data_ptr(), n, 2, 2 if words == 2 else 0), world._h)
    world.wait()
    order = np.lexsort(keys[::-1]) if words == 2 else np.argsort(keys[0], kind="stable")
    assert np.array_equal(payload.cpu().numpy(), order)
    for got, want in zip(tensors, keys):
        assert np.array_equal(got.cpu().numpy(), want[order])
    world.close()


def test_three_grid_runs_of_uneven_size_share_a_sort():
    # 2,500 boxes asleep (more than one tile of entries), a hundred woken, the floor immovable
    scene = scenes.resting_field(50)
    world = World()
    ids = scene.build(world)
    oracle = oracle_from_world(world, DT)
    for step in range(70):
        if step == 60:
            edits = np.concatenate([R.body_edit(R.EDIT_IMPULSE, velocity=(0.0, 3000.0, 0.0))] * 100)
            world.edit_bodies(ids[:100], edits)
            oracle.edit_bodies(ids[:100], edits)
        world.step(DT)
        oracle.step(DT)
        if step >= 58:
            world.wait()
            compare_step(world, oracle, step)
    world.close()


def query_mix(world):
    """Every kind, from a few candidates to more than a warp holds (none past the limit)."""
    at = world.read_states()["position"][:-1]
    centre = np.median(at, axis=0)
    quat = np.array([0.1, -0.4, 0.2, 0.88])
    quat /= np.linalg.norm(quat)
    box, ball = dict(kind=R.SHAPE_CUBOID, half_extents=(1.2, 0.4, 0.8)), dict(kind=R.SHAPE_SPHERE, radius=0.4)
    all_hits = R.query_filter(max_hits=4096)
    queries = [R.sphere_query(centre, float(r), all_hits) for r in (0.3, 1.5, 3.0, 3.6)]
    queries += [R.ray_query((x, 40.0, z), (0.0, -1.0, 0.0), 60.0, R.query_filter(max_hits=64)) for x, _, z in at[::200]]
    queries += [R.ray_query(centre - (30.0, 0.0, 20.0), (30.0, 0.2, 20.0), 80.0, R.query_filter(max_hits=64))]
    queries += [R.overlap_query(box, quat, p, R.query_filter(max_hits=32)) for p in at[::400]]
    queries += [R.overlap_query(dict(kind=R.SHAPE_CUBOID, half_extents=(2.0, 1.5, 2.0)), quat, centre, all_hits)]
    queries += [R.sweep_query(ball, quat, p + (0.0, 6.0, 0.0), (0.3, -1.0, 0.1), 12.0, R.query_filter(max_hits=8)) for p in at[::500]]
    queries += [R.point_query(at[7]), R.cuboid_query(at[11], (0.3, 0.3, 0.3))]
    return queries


@pytest.fixture(scope="module")
def query_world():
    world = World()
    scenes.mixed_pile(14, seed=2).build(world)
    for _ in range(90):
        world.step(DT)
    world.wait()
    queries = query_mix(world)
    small, hits = compare_queries(world, queries)  # against the oracle
    assert world.debug_paths()["block_queries"] == len(queries)
    yield world, np.concatenate(queries), small, hits
    world.close()


@pytest.mark.parametrize("per_sm", [1, 3, 9])
def test_query_batches_on_both_sides_of_the_lines(query_world, per_sm):
    # the same queries again and again, up to per_sm of them an SM: blocks, then warps that hand on the
    # wide ones, then warps that hand on only what they cannot hold
    world, mix, small, hits = query_world
    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    pick = np.arange(n) % len(mix)
    got, got_hits = world.query(mix[pick])
    paths = world.debug_paths()
    if per_sm == 1:
        assert paths["warp_queries"] == 0
    elif per_sm == 3:
        assert 0 < paths["warp_queries"] < n // 2
    else:
        assert n // 2 < paths["warp_queries"] < n
    for name in ("count", "overflow"):
        assert np.array_equal(got[name], small[name][pick]), name
    for i, j in enumerate(pick):
        one = got_hits[got["hit_base"][i]: got["hit_base"][i] + got["count"][i]]
        want = hits[small["hit_base"][j]: small["hit_base"][j] + small["count"][j]]
        assert one.tobytes() == want.tobytes(), f"query {i}"


@pytest.mark.parametrize("copies", [1, 500])
def test_a_query_past_the_candidate_limit_is_flagged(query_world, copies):
    # a box over most of the pile meets more than the 4,096 entries a query takes
    world, mix = query_world[0], query_world[1]
    centre = mix["origin"][0]
    got, _ = world.query(np.concatenate([R.sphere_query(centre, 6.0, R.query_filter(max_hits=8))] * copies))
    assert np.all(got["overflow"] == 1) and np.all(got["count"] == 8)
    assert world.debug_paths()["block_queries"] == copies


def test_a_restored_world_repeats_its_steps_with_most_of_the_stream_empty():
    world = World(capacity={"contacts": 1 << 18})
    scenes.mixed_pile(8, seed=4).build(world)
    for _ in range(60):
        world.step(DT)
    snapshot = world.snapshot()
    runs = []
    for _ in range(2):
        world.restore(snapshot)
        for _ in range(5):
            world.step(DT)
        world.wait()
        runs.append((world.read_states(), world.debug_contacts()))
    assert runs[0][0].tobytes() == runs[1][0].tobytes()
    assert runs[0][1].tobytes() == runs[1][1].tobytes()
    world.close()
