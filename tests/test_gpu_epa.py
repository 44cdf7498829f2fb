"""EPA of deep overlaps against the oracle, one shape-kind combination at a time: polytopes of a
few faces (boxes, cones) up to those of smooth shapes, whose fans and horizons are the widest and
whose vertices run out last.  Tolerance: that of the pair query tests (1e-4 of max(1, |x|); both
sides evaluate the same FP32 / FP64 arithmetic, so nearly every pair is equal to the bit)."""
import numpy as np
import pytest

import oracle_lib as O
from jitterphysics2_gb300 import abi, scenes
from jitterphysics2_gb300.world import world_for_scene

pytestmark = pytest.mark.gpu

KINDS = [abi.SHAPE_BOX, abi.SHAPE_SPHERE, abi.SHAPE_CAPSULE, abi.SHAPE_CYLINDER, abi.SHAPE_CONE, abi.SHAPE_POINTCLOUD]


def overlapping(kind, seed, n=40):
    """Bodies of one kind, and of every kind, packed around the origin."""
    sc = scenes.free_cluster(n=12 * n, seed=seed)
    kinds = sc["shapes"]["kind"]
    first = np.nonzero(kinds == kind)[0][:n]
    rng = np.random.default_rng(seed)
    sc["bodies"]["position"] = rng.uniform(-0.25, 0.25, (len(kinds), 3)).astype(np.float32)
    other = rng.integers(0, len(kinds), len(first))
    pairs = np.array([(min(a, b), max(a, b)) for a, b in zip(first, other) if a != b], np.int32)
    return sc, pairs


@pytest.mark.parametrize("kind", KINDS)
def test_deep_pairs_match_the_oracle(kind):
    sc, pairs = overlapping(kind, seed=31 + kind)
    w = world_for_scene(sc)
    hit, pa, pb, n, depth = w.collide_pairs(pairs)
    o = O.OracleWorld(sc)
    want = [o.collide(int(a), int(b)) for a, b in pairs]
    assert [bool(h) for h in hit] == [bool(r[0]) for r in want]
    deep = np.array([r[4] > 0.02 for r in want]) & hit
    assert deep.sum() > len(pairs) // 2
    got = np.concatenate([pa, pb, n, depth[:, None]], 1)[deep].astype(np.float64)
    ref = np.array([np.concatenate([r[1], r[2], r[3], [r[4]]]) for r in want])[deep]
    err = np.abs(got - ref).max(1) / np.maximum(1.0, np.abs(ref).max(1))
    assert (err < 1e-4).all(), (np.sort(err)[-5:], pairs[deep][np.argsort(err)[-5:]])


@pytest.mark.parametrize("kind", KINDS)
def test_deep_pairs_equal_the_oracle_to_the_bit(kind):
    # the same FP32 and FP64 operations in the same order on both sides, none of them fused; a wrong lane,
    # sign or constant of the face geometry shows in the last bits long before it shows at 1e-4
    sc, pairs = overlapping(kind, seed=61 + kind, n=120)
    w = world_for_scene(sc)
    hit, pa, pb, n, depth = w.collide_pairs(pairs)
    o = O.OracleWorld(sc)
    want = [o.collide(int(a), int(b)) for a, b in pairs]
    got = np.concatenate([pa, pb, n, depth[:, None]], 1)[hit]
    ref = np.array([np.concatenate([r[1], r[2], r[3], [r[4]]]) for r in want], np.float32)[hit]
    assert len(got) > len(pairs) // 2
    assert (got == ref).all(1).mean() >= 0.99
