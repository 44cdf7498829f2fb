"""Fewer bodies uploaded than before, with the constraints (and, without new shapes, the shapes and
contacts) of the others still there: those rows keep being solved against the bodies as they were
last, step after step, and the order keys stay a valid order (rows with one key share no dynamic
body)."""
import numpy as np
import pytest

from jitterphysics2_gb300 import abi, scenes
from jitterphysics2_gb300.world import world_for_scene

pytestmark = pytest.mark.gpu


def limbs():
    sc = scenes.limb_chains(n_chains=6, links=5)
    return sc, len(sc["bodies"]) - 3  # the last three links of the last chain


def pile():
    sc = scenes.mixed_pile(n=60, box=(6.0, 6.0, 6.0), y0=-2.5, cells=6, seed=3, lattice=1.5)
    return sc, len(sc["bodies"]) - 10


def assert_valid_order(keys, b1, b2, dynamic):
    """No dynamic body twice under one key."""
    seen = set()
    for key, pair in zip(keys.tolist(), zip(b1.tolist(), b2.tolist())):
        for b in pair:
            if dynamic[b]:
                assert (key, b) not in seen, (key, b)
                seen.add((key, b))


@pytest.mark.parametrize("make", [limbs, pile])
@pytest.mark.parametrize("partitioned", [1, 0])
def test_rows_of_dropped_bodies_stay_in_a_valid_order(make, partitioned):
    sc, keep = make()
    w = world_for_scene(sc, partitioned_solve=partitioned, record_residual=1)
    for _ in range(30):
        w.step(sc["dt"])
    w.set_bodies(w.bodies()[:keep])
    dynamic = sc["bodies"]["motion_type"] == abi.MOTION_DYNAMIC
    for _ in range(150):  # (more than there are colours: none may be lost from step to step)
        w.step(sc["dt"])
        assert w.counters()["status"] == 0
    c = w.contacts()
    arb = np.unique(c[["color", "body1", "body2"]])
    assert_valid_order(arb["color"], arb["body1"], arb["body2"], dynamic)
    if sc["joints"]:
        j = np.array([(b1, b2) for _, b1, b2, _ in sc["joints"]])
        assert (j >= keep).any()
        assert_valid_order(w.constraints()[0], j[:, 0], j[:, 1], dynamic)
    else:
        assert (c["body2"] >= keep).any() or (c["body1"] >= keep).any()
