"""Mesh-edge records of a step with many colliding records (their manifolds left to threads) against
the same bodies alone (manifolds by warps): the same contacts to the bit."""
import numpy as np
import pytest

from jitterphysics2_gb300 import abi, scenes
from jitterphysics2_gb300.world import world_for_scene

pytestmark = pytest.mark.gpu


def scene(depth, extra):
    """300 spheres and boxes across a heightfield's edges, and `extra` overlapping pairs far away."""
    sc = dict(scenes.mixed_pile(n=10, box=(20.0, 4.0, 20.0), y0=0.0, cells=16, seed=29))
    tris = sc["triangles"]
    rng = np.random.default_rng(11)
    mids = np.concatenate([(tris["a"] + tris["b"]) / 2, (tris["b"] + tris["c"]) / 2, (tris["c"] + tris["a"]) / 2])
    pick = mids[rng.choice(len(mids), 300, replace=False)] + rng.normal(0, 0.01, (300, 3)) * (1, 0, 1)
    cell = np.stack(np.unravel_index(np.arange(extra), (25, 25, 25)), 1) * 4.0 + (100, 50, 100)
    far = np.repeat(cell, 2, 0)
    far[1::2] += (0.0, 0.17, 0.0)
    pos = np.concatenate([pick, far])
    n, nt = len(pos), len(tris)
    bodies = scenes._body(n + 2)
    bodies[:2] = sc["bodies"][:2]
    shapes = np.zeros(1 + nt + n, abi.SHAPE_DTYPE)
    shapes[:1 + nt] = sc["shapes"][:1 + nt]
    for i in range(n):
        si, bi = 1 + nt + i, 2 + i
        sphere = i % 2 == 0
        shapes[si]["body"], shapes[si]["kind"] = bi, abi.SHAPE_SPHERE if sphere else abi.SHAPE_BOX
        shapes[si]["dims"][:3] = 0.1
        bodies["position"][bi] = pos[i] + (0, 0.1 - depth if i < 300 else 0, 0)
        scenes.set_mass(bodies, shapes, np.zeros((0, 3), np.float32), bi, si)
    return dict(sc, bodies=bodies, shapes=shapes, hull=np.zeros((0, 3), np.float32)), 1 + nt + 300


@pytest.mark.parametrize("depth", [0.01, 0.03])
def test_many_and_few_records_agree(depth):
    got = []
    for extra in (0, 8500):
        sc, last = scene(depth, extra)
        w = world_for_scene(sc)
        w.step(sc["dt"])
        assert (w.counters()["colliding"] > 4 * 3 * 4 * 160) == (extra > 0)
        c = w.contacts()
        c = c[(c["shape1"] < last) & (c["shape2"] < last)]
        got.append(c[np.lexsort((c["slot"], c["shape2"], c["shape1"]))])
    assert len(got[0]) > 150
    for f in ("shape1", "shape2", "slot", "usage_mask", "normal", "pos1_local", "pos2_local"):
        assert np.array_equal(got[0][f], got[1][f]), f
