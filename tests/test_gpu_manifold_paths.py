"""Manifolds by warps (few colliding records) and by threads (many): the same pairs of bodies, apart
from each other, in a small and in a large world get the same contacts to the bit."""
import numpy as np
import pytest

from jitterphysics2_gb300 import scenes
from jitterphysics2_gb300.world import world_for_scene

pytestmark = pytest.mark.gpu


def contacts(sc, pairs, shapes=None):
    sc = dict(sc, bodies=sc["bodies"][:2 * pairs], shapes=sc["shapes"][:2 * pairs])
    w = world_for_scene(sc)
    w.step(sc["dt"])
    c = w.contacts()
    c = c[c["shape1"] < 2 * (shapes or pairs)]
    return c[np.lexsort((c["slot"], c["shape2"], c["shape1"]))], w.counters()["colliding"]


@pytest.mark.parametrize("few", [1, 40, 1500])
def test_warps_and_threads_agree(few):
    n = 11000
    sc = scenes.free_cluster(n=2 * n, seed=77)
    rng = np.random.default_rng(78)
    cell = np.stack(np.unravel_index(np.arange(n), (25, 25, 25)), 1) * 8.0
    pos = np.repeat(cell, 2, 0)
    pos[1::2] += rng.normal(0, 0.35, (n, 3))
    sc["bodies"]["position"] = pos.astype(np.float32)
    many, total = contacts(sc, n, few)
    assert total > 4 * 3 * 4 * 160  # more than the warps take on any GPU of this kind
    small, _ = contacts(sc, few)
    assert len(small) > 0
    for f in ("shape1", "shape2", "slot", "usage_mask", "normal", "pos1_local", "pos2_local"):
        assert np.array_equal(small[f], many[f]), f
