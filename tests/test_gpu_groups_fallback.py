"""Rows that belong to no solve group: they send the step to the task solve, so a world steps as
one that records residuals (and so never uses the groups), to the bit."""
import numpy as np
import pytest

from jitterphysics2_gb300 import abi, scenes
from jitterphysics2_gb300.world import World, world_for_scene

pytestmark = pytest.mark.gpu


def pair_of_worlds(sc, **extra):
    return world_for_scene(sc, **extra), world_for_scene(sc, record_residual=1, **extra)


def assert_equal(a, b, joints):
    assert a.counters()["status"] == b.counters()["status"] == 0
    assert np.array_equal(a.bodies(), b.bodies())
    key = ["shape1", "shape2", "slot"]
    ca, cb = (np.sort(w.contacts(), order=key) for w in (a, b))
    assert np.array_equal(ca, cb)
    if joints:
        assert all(np.array_equal(x, y) for x, y in zip(a.constraints(), b.constraints()))


def dynamic_body(sc, world, k):
    """The k-th dynamic body of a world (its first body is the ground)."""
    return int(np.flatnonzero(sc["bodies"]["world"] == world)[1 + k])


@pytest.mark.parametrize("w1,w2", [(0, 1), (0, 39), (39, 2), (17, 5)])
def test_constraint_between_two_worlds(w1, w2):
    sc = scenes.batched_worlds(n_worlds=40, lo=100, hi=130, seed=8)
    b1, b2 = dynamic_body(sc, w1, 3), dynamic_body(sc, w2, 5)
    p = sc["bodies"]["position"]
    sc["joints"] = sc["joints"] + [(abi.CONSTRAINT_BALLSOCKET, b1, b2, tuple((p[b1] + p[b2]) / 2))]
    a, b = pair_of_worlds(sc)
    for _ in range(25):
        a.step(sc["dt"])
        b.step(sc["dt"])
    assert_equal(a, b, True)


@pytest.mark.parametrize("target", [0, 7])
def test_constrained_body_moved_to_another_world_and_back(target):
    sc = scenes.batched_worlds(n_worlds=8, lo=30, hi=60, seed=9)
    i = sc["joints"][0][2]
    home = int(sc["bodies"]["world"][i])
    a, b = pair_of_worlds(sc)
    ha, hb = a.bodies(), b.bodies()
    for world in (home, target if target != home else 3, home):
        for _ in range(8):
            ha["world"][i] = hb["world"][i] = world
            a.step_host(sc["dt"], ha)
            b.step_host(sc["dt"], hb)
        assert_equal(a, b, True)


def test_contact_between_two_of_the_worlds_that_share_a_cell():
    # worlds from 65,535 on share the last cell of the schedule, so that a contact cached before
    # one of its bodies moved from one of them to another stays in a task
    n = 65540
    b = np.zeros(4, abi.BODY_DTYPE)
    b["orientation"][:, 3] = 1.0
    b["position"][:, :2] = (0.0, 0.0), (0.0, 0.99), (5.0, 0.0), (5.0, 0.99)
    b["flags"] = abi.BODY_ACTIVE | abi.BODY_NO_GRAVITY
    b["inv_mass"] = 1.0
    b["inv_inertia"][:, [0, 3, 5]] = 6.0
    b["friction"] = 0.5
    b["linear_damping"] = b["angular_damping"] = 1.0
    b["world"] = (n - 2, n - 2, n - 1, n - 1)
    s = np.zeros(4, abi.SHAPE_DTYPE)
    s["kind"] = abi.SHAPE_BOX
    s["body"] = np.arange(4)
    s["dims"][:, :3] = 0.5
    pair = []
    for residual in (0, 1):
        w = World(max_bodies=n, max_shapes=16, max_pairs=4096, max_arbiters=4096, max_constraints=16, n_worlds=n,
                  allow_deactivation=0, record_residual=residual)
        w.set_bodies(b)
        w.set_shapes(s)
        host = w.bodies()
        for k in range(12):
            if k == 4:
                host["world"][1] = n - 1
            w.step_host(1.0 / 100.0, host)
        pair.append(w)
    assert (pair[1].contacts()["body2"] == 1).any()  # the contact between worlds is still cached
    assert_equal(*pair, False)


@pytest.mark.parametrize("make", [lambda: scenes.limb_chains(n_chains=6, links=5),
                                  lambda: scenes.batched_worlds(n_worlds=6, lo=20, hi=40, seed=5)])
@pytest.mark.parametrize("new_shapes", [True, False])
def test_constraints_of_bodies_beyond_the_uploaded_ones(make, new_shapes):
    # fewer bodies than before: the constraints of the others stay
    sc = make()
    keep = max(max(j[1], j[2]) for j in sc["joints"]) - 1  # (at least two bodies of a constraint are dropped)
    a, b = pair_of_worlds(sc)
    for w in (a, b):
        for _ in range(10):
            w.step(sc["dt"])
        w.set_bodies(w.bodies()[:keep])
        if new_shapes:
            w.set_shapes(sc["shapes"][sc["shapes"]["body"] < keep], sc["hull"], sc["triangles"])
        for _ in range(20):
            w.step(sc["dt"])
    assert_equal(a, b, True)


def test_more_constraints_on_a_body_than_colours():
    # 140 constraints on one body, 128 colours: the step reports it, and no group waits for a row
    n = 140
    b = np.zeros(n + 1, abi.BODY_DTYPE)
    b["orientation"][:, 3] = 1.0
    b["position"][1:, 0] = 2.0 + 1.5 * np.arange(n)
    b["flags"] = abi.BODY_ACTIVE
    b["inv_mass"] = 1.0
    b["inv_inertia"][:, [0, 3, 5]] = 6.0
    b["linear_damping"] = b["angular_damping"] = 1.0
    s = np.zeros(n + 1, abi.SHAPE_DTYPE)
    s["kind"] = abi.SHAPE_BOX
    s["body"] = np.arange(n + 1)
    s["dims"][:, :3] = 0.5
    w = World(max_bodies=n + 1, max_constraints=n, allow_deactivation=0)
    w.set_bodies(b)
    w.set_shapes(s)
    for k in range(100):
        w.add_constraint(abi.CONSTRAINT_BALLSOCKET, 0, k + 1, (1.0, 0.0, 0.0))
    w.step(1.0 / 100.0)
    assert sum(w.solve_groups()) == 1
    for k in range(100, n):
        w.add_constraint(abi.CONSTRAINT_BALLSOCKET, 0, k + 1, (1.0, 0.0, 0.0))
    with pytest.raises(abi.JitterError) as e:
        w.step(1.0 / 100.0)
    assert e.value.code == abi.JG_ERR_CAPACITY
    assert w.solve_groups() == (0, 0, 0)
