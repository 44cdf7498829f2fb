"""Bodies across a heightfield's inner edges at depths on both sides of EPA's threshold (0.02):
shallow ones reach the triangle-edge filter by a rerun with EPA, deep ones with the result EPA
has just returned.  The step's contact cache against the oracle's, with the tolerances of the
heightfield test of the other suites."""
import numpy as np
import pytest

import oracle_lib as O
from jitterphysics2_gb300 import abi, scenes
from jitterphysics2_gb300.world import world_for_scene
from test_gpu_parity import compare_contact_caches

pytestmark = pytest.mark.gpu

KINDS = [(abi.SHAPE_SPHERE, (0.15, 0, 0), 0.15), (abi.SHAPE_BOX, (0.1, 0.1, 0.1), 0.1),
         (abi.SHAPE_CAPSULE, (0.1, 0.1, 0), 0.2), (abi.SHAPE_CYLINDER, (0.12, 0.2, 0), 0.1)]


@pytest.mark.parametrize("depth", [0.01, 0.03, 0.08])
def test_edge_contacts_match_the_oracle(depth):
    sc = dict(scenes.mixed_pile(n=10, box=(20.0, 4.0, 20.0), y0=0.0, cells=16, seed=29))
    tris = sc["triangles"]
    rng = np.random.default_rng(11)
    mids = np.concatenate([(tris["a"] + tris["b"]) / 2, (tris["b"] + tris["c"]) / 2, (tris["c"] + tris["a"]) / 2])
    pick = mids[rng.choice(len(mids), 300, replace=False)] + rng.normal(0, 0.01, (300, 3)) * (1, 0, 1)
    n, nt = len(pick), len(tris)
    bodies = scenes._body(n + 2)
    bodies[:2] = sc["bodies"][:2]
    shapes = np.zeros(1 + nt + n, abi.SHAPE_DTYPE)
    shapes[:1 + nt] = sc["shapes"][:1 + nt]
    for i in range(n):
        kind, dims, rest = KINDS[i % len(KINDS)]
        si, bi = 1 + nt + i, 2 + i
        shapes[si]["body"], shapes[si]["kind"], shapes[si]["dims"][:3] = bi, kind, dims
        bodies["position"][bi] = pick[i] + (0, rest - depth, 0)
        scenes.set_mass(bodies, shapes, np.zeros((0, 3), np.float32), bi, si)
    sc2 = dict(sc, bodies=bodies, shapes=shapes, hull=np.zeros((0, 3), np.float32))
    g = world_for_scene(sc2)
    g.step(sc2["dt"])
    gc = g.contacts()
    o = O.OracleWorld(sc2)
    o.narrowphase()
    oc = o.contacts()
    kinds = sc2["shapes"]["kind"]
    assert sum(kinds[r["shape1"]] == abi.SHAPE_TRIANGLE or kinds[r["shape2"]] == abi.SHAPE_TRIANGLE for r in gc) > 150
    stats = compare_contact_caches(gc, oc)
    assert stats["common_keys"] >= 0.999 * stats["keys"], stats
    assert stats["slot_mismatch"] <= 0.001 * stats["keys"], stats
    assert stats["normal_ok"] >= 0.999 and stats["point_ok"] >= 0.999, stats
