"""The batch-size dispatches and tile edges of the step's kernels, each against its reference.

* The GJK runs a pair on a lane group up to 8,192 pairs and on a lane above that: piles on both
  sides of the line are compared with the oracle, contact for contact.
* The coarse pair walk gives a thread one cell up to 8,192 colliders and a level slice above: fields
  just below and above the line give the oracle's pair list.
* The sorts' tiles hold 4,096 keys, and up to three grid runs share a sort's launches: key counts at
  the tile edges against numpy, and a half-resting world against the oracle.
* A query with more than 512 candidates leaves its warp for a block.
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


@pytest.mark.parametrize("n", [4095, 4096, 4097, 8191, 8192, 8193, 3 * 4096 + 1])
@pytest.mark.parametrize("words", [1, 2])
def test_sort_at_the_tile_edges(n, words):
    rng = np.random.default_rng(n + words)
    # few distinct keys, so that the order of equal ones shows
    keys = rng.integers(0, 700, (words, n), dtype=np.int64).astype(np.int32)
    world = World(capacity={"pairs": 1 << 16})
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


def test_a_query_with_many_candidates_leaves_its_warp():
    world = World()
    scenes.mixed_pile(14, seed=2).build(world)
    for _ in range(90):
        world.step(DT)
    world.wait()
    at = world.read_states()["position"][:-1]
    centre = np.median(at, axis=0)
    # radii whose boxes hold a few dozen, several hundred and more than 512 entries (all below the 4,096 kept), in one batch
    compare_queries(world, [R.sphere_query(centre, float(r), R.query_filter(max_hits=4096)) for r in (0.3, 1.5, 3.0, 3.6)] +
                    [R.ray_query((x, 40.0, z), (0.0, -1.0, 0.0), 60.0, R.query_filter(max_hits=64))
                     for x, _, z in at[::200]] +
                    [R.ray_query(centre - (30.0, 0.0, 20.0), (30.0, 0.2, 20.0), 80.0, R.query_filter(max_hits=64))])
    world.close()


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
