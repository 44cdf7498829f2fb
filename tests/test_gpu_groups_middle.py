"""The group solve of a batch large enough for the launch between the small and the large groups,
against the task solve (a world that records residuals), to the bit: worlds on both sides of
the small and the middle CTA's shared memory."""
import numpy as np
import pytest

from jitterphysics2_gb300 import scenes
from jitterphysics2_gb300.world import world_for_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi", [(8, 24), (24, 300)])
def test_middle_groups_and_tasks_give_the_same_bits(lo, hi):
    sc = scenes.batched_worlds(n_worlds=2600, lo=lo, hi=hi, seed=21)
    a = world_for_scene(sc)
    b = world_for_scene(sc, record_residual=1)
    for _ in range(25):
        a.step(sc["dt"])
        b.step(sc["dt"])
    assert a.counters()["contacts"] == b.counters()["contacts"] > 0
    assert np.array_equal(a.bodies(), b.bodies())
    key = ["shape1", "shape2", "slot"]
    ca, cb = (np.sort(w.contacts(), order=key) for w in (a, b))
    assert np.array_equal(ca, cb)
    assert all(np.array_equal(x, y) for x, y in zip(a.constraints(), b.constraints()))


def test_the_middle_launch_has_groups():
    sc = scenes.batched_worlds(n_worlds=2600, lo=24, hi=300, seed=21)
    a = world_for_scene(sc)
    for _ in range(3):
        a.step(sc["dt"])
        assert all(n > 0 for n in a.solve_groups())
