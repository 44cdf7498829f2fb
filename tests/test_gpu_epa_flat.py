"""EPA where faces degenerate: plates and needles whose polytopes have faces nearly through the
origin or nearly without area, so that the signs of their weights and the reliability of their
normals are decided by the full arithmetic, beside shapes of a hundred times the size.  Against the
oracle, with the tolerance of the pair query tests (1e-4 of max(1, |x|))."""
import numpy as np
import pytest

import oracle_lib as O
from jitterphysics2_gb300 import abi, scenes
from jitterphysics2_gb300.world import world_for_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(2.0, 1e-3, 2.0), (1e-3, 3.0, 1e-3), (200.0, 200.0, 200.0)])
def test_flat_and_large_boxes_match_the_oracle(dims):
    sc = scenes.free_cluster(n=120, seed=5)
    boxes = sc["shapes"]["kind"] == abi.SHAPE_BOX
    sc["shapes"]["dims"][boxes, :3] = dims
    rng = np.random.default_rng(6)
    sc["bodies"]["position"] = rng.uniform(-0.2, 0.2, (120, 3)).astype(np.float32)
    sc["bodies"]["orientation"][::2] = (0.0, 0.0, 0.0, 1.0)  # axis-aligned: exact ties
    i, j = np.triu_indices(120, 1)
    pairs = np.stack([i, j], 1)[boxes[i] | boxes[j]][::3].astype(np.int32)
    w = world_for_scene(sc)
    hit, pa, pb, n, depth = w.collide_pairs(pairs)
    o = O.OracleWorld(sc)
    want = [o.collide(int(a), int(b)) for a, b in pairs]
    assert [bool(h) for h in hit] == [bool(r[0]) for r in want]
    got = np.concatenate([pa, pb, n, depth[:, None]], 1)[hit].astype(np.float64)
    ref = np.array([np.concatenate([r[1], r[2], r[3], [r[4]]]) for r in want])[hit]
    err = np.abs(got - ref).max(1) / np.maximum(1.0, np.abs(ref).max(1))
    assert (err < 1e-4).all(), (np.sort(err)[-5:], pairs[hit][np.argsort(err)[-5:]])


@pytest.mark.parametrize("dims", [(2.0, 1e-3, 2.0), (1e-3, 3.0, 1e-3), (200.0, 200.0, 200.0)])
def test_flat_and_large_boxes_equal_the_oracle_to_the_bit(dims):
    sc = scenes.free_cluster(n=120, seed=15)
    boxes = sc["shapes"]["kind"] == abi.SHAPE_BOX
    sc["shapes"]["dims"][boxes, :3] = dims
    rng = np.random.default_rng(16)
    sc["bodies"]["position"] = rng.uniform(-0.2, 0.2, (120, 3)).astype(np.float32)
    sc["bodies"]["orientation"][::2] = (0.0, 0.0, 0.0, 1.0)  # axis-aligned: exact ties
    i, j = np.triu_indices(120, 1)
    pairs = np.stack([i, j], 1)[boxes[i] | boxes[j]][::3].astype(np.int32)
    w = world_for_scene(sc)
    hit, pa, pb, n, depth = w.collide_pairs(pairs)
    o = O.OracleWorld(sc)
    want = [o.collide(int(a), int(b)) for a, b in pairs]
    got = np.concatenate([pa, pb, n, depth[:, None]], 1)[hit]
    ref = np.array([np.concatenate([r[1], r[2], r[3], [r[4]]]) for r in want], np.float32)[hit]
    assert len(got) > len(pairs) // 2
    assert (got == ref).all(1).mean() >= 0.99
