"""The group solve (one CTA per independent part of the scene) against the task solve.

Recording residuals keeps a world on the task solve, and both solves run the rows of every body
in the same order, so two worlds that differ only in that flag have to stay equal to the
bit: bodies, contacts' impulses and constraints.  The scenes have parts at the edges of the
groups: one row and one body, more rows than threads, components on either side of the row
limit, every constraint kind, batches, static, sleeping and kinematic neighbours."""
import numpy as np
import pytest

from jitterphysics2_gb300 import abi, scenes
from jitterphysics2_gb300.world import world_for_scene

pytestmark = pytest.mark.gpu


def small_pile(n, seed=3):
    width = 1.5 * max(3, round(n ** (1 / 3)))  # on a lattice: a random box of 500 exceeds the pools
    return scenes.mixed_pile(n=n, box=(width, 6.0, width), y0=-2.5, cells=6, seed=seed, lattice=1.5)


def stacks(side, friction=0.6):
    sc = scenes.box_grid(n_side=side, friction=friction)
    sc["bodies"]["position"][1:, 1] = 0.5 + (np.arange(side ** 3) // side) % side
    return sc


def kinematic_floor():
    sc = stacks(3)
    sc["bodies"]["motion_type"][0] = abi.MOTION_KINEMATIC
    sc["bodies"]["velocity"][0] = (0.3, 0.05, 0.0)
    return sc


def gyroscopic_free():
    sc = scenes.free_cluster(n=40, spacing=1.6)
    sc["bodies"]["flags"] |= abi.BODY_GYROSCOPIC
    sc["bodies"]["flags"][::3] |= 1 << abi.BODY_LOCKS_SHIFT  # a locked axis
    return sc


CASES = {
    "one_box": (lambda: stacks(1), 30, {}),
    "two_boxes_wide": (lambda: stacks(2), 30, {}),
    "stacks_7": (lambda: stacks(7), 20, {}),
    "stacks_7_asleep": (lambda: stacks(7), 160, dict(allow_deactivation=1)),
    "pile_below_the_row_limit": (lambda: small_pile(60), 60, {}),
    "pile_above_the_row_limit": (lambda: small_pile(500), 40, {}),
    "kinematic": (kinematic_floor, 20, {}),
    "free_bodies": (gyroscopic_free, 30, {}),
    "limbs": (lambda: scenes.limb_chains(n_chains=37, links=5), 20, {}),
    "mechanisms": (lambda: scenes.mechanism_chains(n_chains=9), 20, {}),
    "servos": (lambda: scenes.servo_chains(n_chains=9), 20, {}),
    "worlds_3": (lambda: scenes.batched_worlds(n_worlds=3), 40, {}),
    "worlds_400": (lambda: scenes.batched_worlds(n_worlds=400, hi=64), 20, {}),
    "worlds_large": (lambda: scenes.batched_worlds(n_worlds=5, lo=400, hi=700), 30, {}),
    "bullets": (lambda: scenes.bullets(n=64), 8, {}),
    "no_relaxation": (lambda: stacks(3), 20, dict(relax_iterations=0, substeps=1)),
}


@pytest.mark.parametrize("name", list(CASES))
def test_groups_and_tasks_give_the_same_bits(name):
    make, steps, extra = CASES[name]
    sc = make()
    a = world_for_scene(sc, **extra)
    b = world_for_scene(sc, record_residual=1, **extra)
    for k in range(steps):
        a.step(sc["dt"])
        b.step(sc["dt"])
        if k % 10 == 9 or k == steps - 1:
            assert a.counters()["contacts"] == b.counters()["contacts"]
            assert np.array_equal(a.bodies(), b.bodies()), (name, k)
    key = ["shape1", "shape2", "slot"]
    ca, cb = (np.sort(w.contacts(), order=key) for w in (a, b))
    assert np.array_equal(ca, cb)
    if sc["joints"]:
        assert all(np.array_equal(x, y) for x, y in zip(a.constraints(), b.constraints()))


@pytest.mark.parametrize("name", [n for n in CASES if n != "kinematic"])
def test_the_groups_solve_these_scenes(name):
    # (otherwise both worlds of the test above run the task solve)
    make, steps, extra = CASES[name]
    sc = make()
    a = world_for_scene(sc, **extra)
    by_tasks = []
    for k in range(steps):
        a.step(sc["dt"])
        if a.counters()["arbiters"] or sc["joints"]:
            asleep = not (a.bodies()["flags"] & abi.BODY_ACTIVE)[sc["bodies"]["motion_type"] == abi.MOTION_DYNAMIC].any()
            if any(a.solve_groups()) == asleep:
                by_tasks.append(k)
    if name == "pile_above_the_row_limit":  # packed at first, then the bodies fall apart
        assert 0 < len(by_tasks) < steps
    else:
        assert not by_tasks


def test_solve_groups_is_zero_after_the_task_solve():
    sc = stacks(3)
    a, b, c = (world_for_scene(sc, **kw) for kw in ({}, dict(record_residual=1), dict(partitioned_solve=0)))
    for w in (a, b, c):
        w.step(sc["dt"])
    assert [sum(w.solve_groups()) for w in (a, b, c)] == [9, 0, 0]
    a.stabilize(sc["dt"], 2)
    assert a.solve_groups() == (0, 0, 0)
    k = world_for_scene(kinematic_floor())
    k.step(sc["dt"])
    assert k.counters()["arbiters"] > 0 and k.solve_groups() == (0, 0, 0)


def row_of(n, kind):
    """n bodies side by side on the floor, each touching its neighbours: one part of up to 2 n - 1 rows."""
    sc = scenes.box_grid(n_side=1, friction=0.6)
    sc["bodies"] = sc["bodies"][[0] + [1] * n].copy()
    sc["shapes"] = sc["shapes"][[0] + [1] * n].copy()
    sc["shapes"]["kind"][1:] = kind
    sc["shapes"]["body"] = np.arange(n + 1)
    sc["bodies"]["position"][1:] = np.stack([0.999 * (np.arange(n) - n / 2), np.full(n, 0.495), np.zeros(n)], 1)
    return sc


def assert_route_and_bits(sc, rows, by_groups):
    a, b = world_for_scene(sc), world_for_scene(sc, record_residual=1)
    for _ in range(5):
        a.step(sc["dt"])
        b.step(sc["dt"])
        assert rows(a.counters())
        assert any(a.solve_groups()) == by_groups
    assert np.array_equal(a.bodies(), b.bodies())
    key = ["shape1", "shape2", "slot"]
    assert np.array_equal(*(np.sort(w.contacts(), order=key) for w in (a, b)))


@pytest.mark.parametrize("n,by_groups", [(160, True), (161, False)])
def test_part_at_the_row_limit(n, by_groups):
    # spheres: one contact to a row, 319 or 321 rows on both sides of the limit of 320
    assert_route_and_bits(row_of(n, abi.SHAPE_SPHERE), lambda c: (c["arbiters"] <= 320) == by_groups, by_groups)


@pytest.mark.parametrize("n,by_groups", [(95, True), (105, False)])
def test_part_at_the_contact_limit(n, by_groups):
    # boxes: four contacts to a row, and no more than 8 n - 4 of them; the limit is 800
    assert_route_and_bits(row_of(n, abi.SHAPE_BOX), lambda c: (c["contacts"] <= 800) == by_groups and c["arbiters"] <= 320, by_groups)


@pytest.mark.parametrize("worlds,by_groups", [(150, True), (160, False), (310, True)])
def test_batch_of_dense_worlds(worlds, by_groups):
    # 64 boxes side by side in each world, some 508 contacts: between the two limits for one and for two groups an SM,
    # and small enough for a small CTA, of which large batches keep eight an SM
    one = row_of(64, abi.SHAPE_BOX)
    n = len(one["bodies"])
    sc = dict(one, n_worlds=worlds, bodies=np.tile(one["bodies"], worlds), shapes=np.tile(one["shapes"], worlds))
    sc["bodies"]["world"] = np.repeat(np.arange(worlds), n)
    sc["shapes"]["body"] = np.arange(n * worlds)
    assert_route_and_bits(sc, lambda c: 350 * worlds < c["contacts"] <= 800 * worlds, by_groups)
