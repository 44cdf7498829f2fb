"""Pair queries on both sides of the sizes at which the query changes from a warp per pair to two
stages, groups the pairs by kind, and splits them over the world's lists: the answer to each pair
is that of the same pair asked for alone in a small batch, to the bit."""
import numpy as np
import pytest

from jitterphysics2_gb300 import scenes
from jitterphysics2_gb300.world import World

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def world():
    sc = scenes.free_cluster(n=150, spacing=1.2)
    w = World(max_bodies=len(sc["bodies"]), max_arbiters=5000, max_pairs=6000)  # lists of 5000: several chunks
    w.set_bodies(sc["bodies"])
    w.set_shapes(sc["shapes"], sc["hull"])
    i, j = np.triu_indices(150, 1)
    near = np.linalg.norm(sc["bodies"]["position"][i] - sc["bodies"]["position"][j], axis=1) < 2.5
    base = np.stack([i[near], j[near]], 1).astype(np.int32)[:1500]
    return w, base, [w.collide_pairs(base[k:k + 300]) for k in range(0, len(base), 300)]


@pytest.mark.parametrize("n", [1, 31, 2433, 5000, 7296, 7297, 9095, 9096, 10000, 10001, 20001])
def test_batch_sizes_agree(world, n):
    w, base, parts = world
    want = [np.concatenate([p[f] for p in parts]) for f in range(5)]
    pick = np.random.default_rng(n).integers(0, len(base), n)
    got = w.collide_pairs(base[pick])
    assert want[0].any() and not want[0].all()
    for f in range(5):
        assert np.array_equal(got[f], want[f][pick])


@pytest.mark.parametrize("lists", [1024, 6667, 6666, 7297, 8000])
def test_small_lists_agree(world, lists):
    # lists of up to 7,296 pairs and more than three chunks: one launch; else chunks of two stages
    w, base, parts = world
    want = [np.concatenate([p[f] for p in parts]) for f in range(5)]
    sc = scenes.free_cluster(n=150, spacing=1.2)
    small = World(max_bodies=len(sc["bodies"]), max_arbiters=lists, max_pairs=lists)
    small.set_bodies(sc["bodies"])
    small.set_shapes(sc["shapes"], sc["hull"])
    pick = np.random.default_rng(lists).integers(0, len(base), 20001)
    got = small.collide_pairs(base[pick])
    for f in range(5):
        assert np.array_equal(got[f], want[f][pick])


def test_batch_sizes_agree_where_a_pose_has_overflowed():
    # a body thrown out of the float range: its queries miss, and the points they report are the same in every batch
    sc = scenes.free_cluster(n=60, spacing=1.2)
    lost = 7
    sc["bodies"]["velocity"][lost] = 3e38
    w = World(max_bodies=60, max_pairs=30000, max_arbiters=30000, gravity=(0.0, 0.0, 0.0), allow_deactivation=0)
    w.set_bodies(sc["bodies"])
    w.set_shapes(sc["shapes"], sc["hull"])
    w.step(1.0)
    w.step(1.0)
    assert not np.isfinite(w.bodies()["position"][lost]).all()
    other = np.delete(np.arange(60), lost)
    base = np.concatenate([np.stack([other, np.full(59, lost)], 1), np.stack([np.full(59, lost), other], 1)]).astype(np.int32)
    alone = w.collide_pairs(base)
    pick = np.random.default_rng(3).integers(0, len(base), 9000)
    got = w.collide_pairs(base[pick])
    for f in range(5):
        assert np.array_equal(got[f], alone[f][pick], equal_nan=f > 0)
