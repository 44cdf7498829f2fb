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
