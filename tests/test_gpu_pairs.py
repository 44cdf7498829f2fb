"""The broadphase's pair list against an all-pairs reference, on both sides of the size at which
the search changes from every box against every box to the tree, and at the edges of the box tiles:
single and batched worlds, every motion type, sleeping bodies, two shapes on one body."""
import numpy as np
import pytest

from jitterphysics2_gb300 import abi
from jitterphysics2_gb300.world import World

pytestmark = pytest.mark.gpu


def spheres(n, n_worlds, seed):
    rng = np.random.default_rng(seed)
    b = np.zeros(n, abi.BODY_DTYPE)
    b["orientation"][:, 3] = 1.0
    b["position"] = rng.uniform(0, max(2.0, 1.1 * n ** (1 / 3)), (n, 3)).astype(np.float32)
    b["motion_type"] = rng.choice([abi.MOTION_DYNAMIC, abi.MOTION_KINEMATIC, abi.MOTION_STATIC], n, p=[0.8, 0.1, 0.1])
    b["flags"] = np.where(rng.random(n) < 0.7, abi.BODY_ACTIVE, 0) | abi.BODY_NO_GRAVITY
    b["inv_mass"] = np.where(b["motion_type"] == abi.MOTION_DYNAMIC, 1.0, 0.0)
    b["inv_inertia"][:, [0, 3, 5]] = b["inv_mass"][:, None]
    b["linear_damping"] = b["angular_damping"] = 1.0
    b["world"] = rng.integers(0, n_worlds, n)
    s = np.zeros(n, abi.SHAPE_DTYPE)
    s["kind"] = abi.SHAPE_SPHERE
    s["body"] = np.where(rng.random(n) < 0.05, np.maximum(np.arange(n) - 1, 0), np.arange(n))
    s["dims"][:, 0] = rng.uniform(0.2, 0.8, n).astype(np.float32)
    return b, s


def reference(b, s):
    r = s["dims"][:, :1]
    p = b["position"][s["body"]]
    lo, hi = p - r, p + r
    body, world = s["body"], b["world"][s["body"]]
    dyn = b["motion_type"][body] == abi.MOTION_DYNAMIC
    act = (b["flags"][body] & abi.BODY_ACTIVE) != 0
    out = []
    for i in range(0, len(s), 256):
        k = slice(i, min(i + 256, len(s)))
        hit = np.ones((k.stop - i, len(s)), bool)
        for c in range(3):
            hit &= ~((hi[k, c, None] < lo[None, :, c]) | (lo[k, c, None] > hi[None, :, c]))
        hit &= (body[k, None] != body) & (world[k, None] == world) & (dyn[k, None] | dyn) & (act[k, None] | act)
        a, c = np.nonzero(hit)
        out.append(np.stack([a + i, c], 1)[a + i < c])
    return np.concatenate(out)


@pytest.mark.parametrize("n,n_worlds", [(2, 1), (127, 1), (128, 1), (129, 2), (1000, 1), (4097, 3), (16384, 1), (16385, 1), (16500, 2)])
def test_pairs_match_all_pairs(n, n_worlds):
    b, s = spheres(n, n_worlds, seed=n)
    w = World(max_bodies=n, max_shapes=n, n_worlds=n_worlds, allow_deactivation=0)
    w.set_bodies(b)
    w.set_shapes(s)
    w.step(1.0 / 100.0)
    got = w.pairs()
    want = reference(b, s)
    assert len(got) == len(want) == w.counters()["pairs"]
    assert np.array_equal(got[np.lexsort(got.T[::-1])], want[np.lexsort(want.T[::-1])])


def rods(n, n_worlds, seed):
    """Parallel thin rods along (1, 1, 1), close together without touching: every two boxes overlap,
    a 128 x 128 tile of them is 16,384 pairs."""
    b, s = spheres(n, n_worlds, seed)
    d = np.array([1.0, 1.0, 1.0]) / np.sqrt(3.0)
    u = np.array([1.0, -1.0, 0.0]) / np.sqrt(2.0)
    v = np.cross(d, u)
    side = int(np.ceil(np.sqrt(n)))
    i = np.arange(n)
    g = np.stack([i % side, i // side], 1) / side - 0.5
    b["position"] = 0.5 * (g[:, :1] * u + g[:, 1:] * v)
    axis = np.cross([0.0, 1.0, 0.0], d)  # turns the capsule's y axis to d
    q = np.append(axis, 1.0 + d[1])
    b["orientation"] = q / np.linalg.norm(q)
    s["kind"] = abi.SHAPE_CAPSULE
    s["body"] = i
    s["dims"][:, 0] = 1e-3
    s["dims"][:, 1] = 2.0
    return b, s


def all_pairs(b, s):
    world, dyn = b["world"][s["body"]], b["motion_type"][s["body"]] == abi.MOTION_DYNAMIC
    act = (b["flags"][s["body"]] & abi.BODY_ACTIVE) != 0
    i, j = np.triu_indices(len(s), 1)
    keep = (world[i] == world[j]) & (dyn[i] | dyn[j]) & (act[i] | act[j])
    return np.stack([i[keep], j[keep]], 1)


@pytest.mark.parametrize("n,n_worlds", [(128, 1), (300, 2), (1000, 1), (4500, 1)])
def test_dense_pairs_match_all_pairs(n, n_worlds):
    # more pairs than a block's buffer holds, in one tile (up to 1,000) and over the tiles of a block (4,500)
    b, s = rods(n, n_worlds, seed=n)
    want = all_pairs(b, s)
    w = World(max_bodies=n, max_shapes=n, max_pairs=len(want) + 1, n_worlds=n_worlds, allow_deactivation=0)
    w.set_bodies(b)
    w.set_shapes(s)
    w.step(1.0 / 100.0)
    got = w.pairs()
    assert len(got) == len(want) == w.counters()["pairs"]
    assert np.array_equal(got[np.lexsort(got.T[::-1])], want)


def test_dense_pairs_beyond_the_pool():
    b, s = rods(1000, 1, seed=1000)
    want = all_pairs(b, s)
    cap = len(want) // 4
    w = World(max_bodies=1000, max_shapes=1000, max_pairs=cap, allow_deactivation=0)
    w.set_bodies(b)
    w.set_shapes(s)
    with pytest.raises(abi.JitterError) as e:
        w.step(1.0 / 100.0)
    assert e.value.code == abi.JG_ERR_CAPACITY
    got = w.pairs()
    assert len(got) == cap
    n = len(s)
    key = np.sort(got[:, 0].astype(np.int64) * n + got[:, 1])
    assert (np.diff(key) > 0).all() and np.isin(key, want[:, 0] * n + want[:, 1]).all()
