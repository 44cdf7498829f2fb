"""Performance cases: what a user of the contact pipeline has it do, through `World`.

A case steps one formed scene (World.step_host: bodies in from pinned host memory, one step,
bodies back), queries shape pairs (World.collide_pairs) or takes the gradients of the learned
warm start (World.mlp_gradients).  The scenes are the package's own workloads (box grid, mixed
pile on a heightfield, towers and rubble, batched worlds, limb chains) at sizes from a handful of
bodies to the largest of each; a scene starts loosely packed and is stepped until its bodies have
landed and its contact cache is filled.
"""
import functools

import numpy as np
import torch

from jitterphysics2_gb300 import abi, learned, scenes
from jitterphysics2_gb300.world import World, world_for_scene

SPACING = 1.6  # of mixed bodies before they settle: few overlaps, a short fall


def listed():
    return [
        # the smallest useful scene, a few stacks on a floor: latency and launches
        {"name": "boxes_27", "kind": "boxes", "side": 3, "substeps": 4, "iterations": 8, "sleep": False},
        # the reference's own benchmark size: a thousand boxes in stacks
        {"name": "boxes_1000", "kind": "boxes", "side": 10, "substeps": 4, "iterations": 8, "sleep": False},
        # a level whose props come to rest, with deactivation on as World has it by default
        {"name": "boxes_resting", "kind": "boxes", "side": 16, "substeps": 4, "iterations": 8, "sleep": True},
        # an ordinary game scene on terrain at World's default solver settings
        {"name": "pile_700", "kind": "pile", "n": 700, "substeps": 1, "iterations": 6, "sleep": False},
        # the narrowphase workload: mixed shapes on a triangle mesh
        {"name": "pile_20k", "kind": "pile", "n": 20000, "substeps": 4, "iterations": 8, "sleep": False},
        # the headline workload
        {"name": "pile_100k", "kind": "pile", "n": 100000, "substeps": 4, "iterations": 8, "sleep": False},
        # a wide scene: tall stacks in thinly spread rubble
        {"name": "towers_50k", "kind": "towers", "towers": 50, "height": 20, "rubble": 49000},
        # independent small scenes stepped as one batch, some with jointed chains: a few, and many
        {"name": "worlds_48", "kind": "worlds", "worlds": 48},
        {"name": "worlds_4096", "kind": "worlds", "worlds": 4096},
        # ragdoll limbs: constraints without contacts
        {"name": "chains_1024", "kind": "chains", "chains": 1024, "links": 6},
        # overlap queries on chosen pairs of shapes
        {"name": "query_30001", "kind": "query", "pairs": 30001},
        # one training batch of the learned warm start
        {"name": "mlp_4096", "kind": "mlp", "samples": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["boxes", "pile", "pile", "towers", "worlds", "chains", "query", "mlp"])
    if kind == "boxes":
        return {"kind": kind, "side": _log_int(rng, 2, 20), "substeps": rng.choice([1, 2, 4]),
                "iterations": rng.randint(4, 10), "sleep": rng.random() < 0.25}
    if kind == "pile":
        return {"kind": kind, "n": _log_int(rng, 60, 90000), "substeps": rng.choice([1, 2, 4]),
                "iterations": rng.randint(4, 10), "sleep": False}
    if kind == "towers":
        return {"kind": kind, "towers": _log_int(rng, 2, 60), "height": rng.randint(5, 24),
                "rubble": _log_int(rng, 300, 48000)}
    if kind == "worlds":
        return {"kind": kind, "worlds": _log_int(rng, 2, 2500)}
    if kind == "chains":
        return {"kind": kind, "chains": _log_int(rng, 3, 1500), "links": rng.randint(3, 9)}
    if kind == "query":
        return {"kind": kind, "pairs": _log_int(rng, 1, 200000)}
    return {"kind": kind, "samples": _log_int(rng, 16, 60000)}


# ---- scenes ------------------------------------------------------------------------------

@functools.lru_cache(maxsize=1)
def _palette():
    """Mixed bodies with their shapes and mass properties, as the package's workloads draw them."""
    sc = scenes.towers_rubble(n_towers=1, height=1, n_rubble=240)
    return sc["bodies"][2:], sc["shapes"][2:], sc["hull"]


@functools.lru_cache(maxsize=8)
def _terrain(cells, extent, amplitude):
    return scenes.heightfield(cells, extent, amplitude)


@functools.lru_cache(maxsize=1)
def _world_templates():
    """A batch of worlds split into its worlds: (bodies, shapes, joints) with local indices."""
    sc = scenes.batched_worlds(n_worlds=32)
    first = np.flatnonzero(np.diff(sc["bodies"]["world"], prepend=-1))
    last = np.append(first[1:], len(sc["bodies"]))
    joints = [[] for _ in first]
    for kind, b1, b2, init in sc["joints"]:
        t = int(sc["bodies"]["world"][b1])
        joints[t].append((kind, b1 - int(first[t]), b2 - int(first[t]), init))
    out = []
    for t, (a, b) in enumerate(zip(first, last)):
        s = sc["shapes"][a:b].copy()
        s["body"] -= a
        out.append((sc["bodies"][a:b], s, joints[t]))
    return out, sc["hull"]


def _mixed(rng, n):
    """n bodies and shapes drawn from the palette, at random orientations."""
    pb, ps, hull = _palette()
    pick = rng.integers(0, len(pb), n)
    bodies, shapes = pb[pick].copy(), ps[pick].copy()
    bodies["orientation"] = scenes.random_quaternions(rng, n)
    return bodies, shapes, hull


def _boxes(case, rng):
    side = case["side"]
    sc = scenes.box_grid(n_side=side, seed=int(rng.integers(1 << 30)))
    level = (np.arange(side ** 3) // side) % side
    sc["bodies"]["position"][1:, 1] = 0.5 + level  # stacked, each on the one below
    return sc


def _pile(case, rng):
    n = case["n"]
    extent = 1.9 * n ** 0.36  # deeper the larger, as heaps are (120 wide at 100,000)
    cells = int(np.clip(round(extent), 4, 64))
    amplitude = min(2.0, extent / 20)
    tris = _terrain(cells, extent, amplitude)
    nt = len(tris)
    mixed, recs, hull = _mixed(rng, n)
    bodies = np.zeros(n + 2, abi.BODY_DTYPE)
    bodies[:2] = mixed[0]
    bodies[2:] = mixed
    shapes = np.zeros(n + 1 + nt, abi.SHAPE_DTYPE)
    scenes.ground(bodies, shapes, 0, 0, size=(3 * extent + 100, 1.0, 3 * extent + 100))
    bodies["position"][1] = 0.0  # the terrain
    bodies["motion_type"][1] = abi.MOTION_STATIC
    bodies["inv_mass"][1] = 0.0
    bodies["inv_inertia"][1] = 0.0
    bodies["orientation"][:2] = (0.0, 0.0, 0.0, 1.0)
    shapes["kind"][1:1 + nt] = abi.SHAPE_TRIANGLE
    shapes["body"][1:1 + nt] = 1
    shapes["data_offset"][1:1 + nt] = np.arange(nt)
    shapes[1 + nt:] = recs
    shapes["body"][1 + nt:] = np.arange(2, n + 2)
    row = max(1, int(extent / SPACING))
    i = np.arange(n)
    pos = np.stack([i % row, i // (row * row), (i // row) % row], 1) * SPACING
    pos[:, [0, 2]] -= (row - 1) * SPACING / 2
    pos += rng.uniform(-0.1, 0.1, pos.shape)
    k = 6 * np.pi / extent  # the height under each column (scenes.heightfield)
    pos[:, 1] += 2.9 + amplitude * np.sin(k * pos[:, 0]) * np.cos(k * pos[:, 2])
    bodies["position"][2:] = pos
    bodies["friction"] = 0.6
    return dict(bodies=bodies, shapes=shapes, hull=hull, triangles=tris, joints=[], dt=1.0 / 100.0, params={})


def _towers(case, rng):
    nt, height, nr = case["towers"], case["height"], case["rubble"]
    side = int(np.ceil(np.sqrt(nt)))
    area = max(float(np.sqrt(nr / 1.9)), 4.0 * side)
    mixed, recs, hull = _mixed(rng, nr)
    tower = scenes.box_grid(n_side=1)["bodies"][1]
    nbox = nt * height
    bodies = np.zeros(1 + nbox + nr, abi.BODY_DTYPE)
    bodies[:1 + nbox] = tower
    bodies[1 + nbox:] = mixed
    shapes = np.zeros(1 + nbox + nr, abi.SHAPE_DTYPE)
    scenes.ground(bodies, shapes, 0, 0, size=(3 * area, 1.0, 3 * area))
    t = np.arange(nbox)
    tx, tz = (t // height) % side, (t // height) // side
    cell = area / side
    bodies["position"][1:1 + nbox] = np.stack([(tx - (side - 1) / 2) * cell, 0.5 + t % height,
                                               (tz - (side - 1) / 2) * cell], 1)
    shapes["kind"][:1 + nbox] = abi.SHAPE_BOX
    shapes["dims"][1:1 + nbox, :3] = 0.5
    shapes[1 + nbox:] = recs
    shapes["body"] = np.arange(1 + nbox + nr)
    # rubble in layers around the towers
    row = int(area / SPACING) + 1
    g = np.arange(row * row)
    xz = np.stack([g % row, g // row], 1) * SPACING - (row - 1) * SPACING / 2
    near = np.abs((xz + area / 2) % cell - cell / 2).max(1)
    free = xz[near > 1.8] if (near > 1.8).any() else xz
    i = np.arange(nr)
    pos = np.stack([free[i % len(free), 0], 0.8 + SPACING * (i // len(free)), free[i % len(free), 1]], 1)
    bodies["position"][1 + nbox:] = pos + rng.uniform(-0.1, 0.1, pos.shape)
    bodies["friction"] = 0.6
    return dict(bodies=bodies, shapes=shapes, hull=hull, triangles=np.zeros(0, abi.TRIANGLE_DTYPE), joints=[],
                dt=1.0 / 100.0, params=dict(substeps=4, solver_iterations=8, relax_iterations=4))


def _worlds(case, rng):
    templates, hull = _world_templates()
    bodies, shapes, joints, base = [], [], [], 0
    for k in range(case["worlds"]):
        b, s, js = templates[(k + case["worlds"]) % len(templates)]
        s = s.copy()
        s["body"] += base
        bodies.append(b)
        shapes.append(s)
        joints += [(kind, base + b1, base + b2, init) for kind, b1, b2, init in js]
        base += len(b)
    world = np.repeat(np.arange(len(bodies)), [len(b) for b in bodies])
    bodies, shapes = np.concatenate(bodies), np.concatenate(shapes)
    bodies["world"] = world
    linked = np.zeros(len(bodies), bool)
    linked[[b for j in joints for b in j[1:3]]] = True
    loose = (bodies["motion_type"] == abi.MOTION_DYNAMIC) & ~linked
    n = int(loose.sum())
    bodies["orientation"][loose] = scenes.random_quaternions(rng, n)
    bodies["position"][loose] += rng.uniform(-0.05, 0.05, (n, 3)).astype(np.float32)
    return dict(bodies=bodies, shapes=shapes, hull=hull, triangles=np.zeros(0, abi.TRIANGLE_DTYPE), joints=joints,
                n_worlds=case["worlds"], dt=1.0 / 120.0,
                params=dict(substeps=4, solver_iterations=8, relax_iterations=4))


SETTLE = {"boxes": 20, "pile": 160, "towers": 120, "worlds": 120, "chains": 20}  # steps before the first pass


def _step_scene(case, rng):
    if case["kind"] == "boxes":
        return _boxes(case, rng)
    if case["kind"] == "pile":
        return _pile(case, rng)
    if case["kind"] == "towers":
        return _towers(case, rng)
    if case["kind"] == "worlds":
        return _worlds(case, rng)
    return scenes.limb_chains(n_chains=case["chains"], links=case["links"], seed=int(rng.integers(1 << 30)))


# ---- states ------------------------------------------------------------------------------

def _pinned(array):
    flat = torch.empty(array.nbytes, dtype=torch.uint8, pin_memory=True).numpy()
    out = flat.view(array.dtype)
    out[:] = array
    return out


def _mlp_data(case, seed):
    rng = np.random.default_rng(seed)
    X = rng.normal(0, 2, (case["samples"], abi.MLP_IN)).astype(np.float32)
    T = rng.normal(0, 3, (case["samples"], abi.MLP_OUT)).astype(np.float32)
    ref = np.random.default_rng(1)
    p = learned.init_params(ref.normal(0, 2, (256, abi.MLP_IN)), ref.normal(0, 3, (256, abi.MLP_OUT)), seed=seed)
    return X, T, p


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        X, T, p = _mlp_data(case, seed)
        w = World(max_bodies=16)
        w.mlp_load(p)
        return {"kind": kind, "world": w, "X": X, "T": T}
    rng = np.random.default_rng(seed)
    if kind == "query":
        # neighbours and near neighbours on a packed lattice: from deep overlaps to clear misses
        side = int(np.clip(round(np.cbrt(case["pairs"] / 4)), 2, 24))  # (at the density of a pile)
        i = np.arange(side ** 3)
        bodies, shapes, hull = _mixed(rng, len(i))
        cell = np.stack([i % side, (i // side) % side, i // (side * side)], 1)
        bodies["position"] = cell * 1.35 + rng.uniform(-0.3, 0.3, cell.shape)
        shapes["body"] = i
        a = rng.integers(0, len(i), case["pairs"])
        step = rng.integers(-1, 2, (case["pairs"], 3))
        step[(step == 0).all(1)] = (0, 1, 0)
        to = cell[a] + step
        to = np.where((to < 0) | (to >= side), cell[a] - step, to)
        b = to[:, 0] + side * (to[:, 1] + side * to[:, 2])
        w = World(max_bodies=len(i), allow_deactivation=0)
        w.set_bodies(bodies)
        w.set_shapes(shapes, hull)
        return {"kind": kind, "world": w, "pairs": np.stack([a, b], 1).astype(np.int32)}
    scene = _step_scene(case, rng)
    extra = {"allow_deactivation": 1} if case.get("sleep") else {}
    if "substeps" in case:
        extra.update(substeps=case["substeps"], solver_iterations=case["iterations"], relax_iterations=4)
    w = world_for_scene(scene, **extra)
    for _ in range(SETTLE[kind]):
        w.step(scene["dt"])
    return {"kind": kind, "world": w, "dt": scene["dt"], "bodies": _pinned(w.bodies())}


def run(state):
    w = state["world"]
    if state["kind"] == "mlp":
        grads, loss = w.mlp_gradients(state["X"], state["T"])
        return {"gradients": grads, "loss": np.float32(loss)}
    if state["kind"] == "query":
        hit, a, b, normal, depth = w.collide_pairs(state["pairs"])
        return {"hit": hit, "point_a": a, "point_b": b, "normal": normal, "depth": depth}
    bodies = state["bodies"]
    w.step_host(state["dt"], bodies)
    out = {f: bodies[f] for f in ("position", "orientation", "velocity", "angular_velocity")}
    seen = w.counters()
    out.update((k, seen[k]) for k in ("pairs", "arbiters", "contacts"))
    return out


# ---- work and exact values -----------------------------------------------------------------

# contact points per body of each scene once it has formed (measured on the workloads)
CONTACTS = {"boxes": 4.0, "pile": 2.6, "towers": 1.7, "worlds": 2.3, "chains": 0.0}


def work(case):
    kind = case["kind"]
    if kind == "mlp":
        n, h, i, o = case["samples"], abi.MLP_HID, abi.MLP_IN, abi.MLP_OUT
        return {"bytes": 4 * (n * (i + o) + 2 * abi.MLP_NW), "flops": 2 * n * (3 * (i * h + h * h + h * o) - i * h)}
    if kind == "query":
        # two bodies' poses and shapes, the pair and its result; about ten support evaluations
        return {"bytes": case["pairs"] * (2 * (32 + 48) + 8 + 44), "flops": case["pairs"] * 10 * 250}
    if kind == "boxes":
        n, joints = case["side"] ** 3, 0
    elif kind == "pile":
        n, joints = case["n"], 0
    elif kind == "towers":
        n, joints = case["towers"] * case["height"] + case["rubble"], 0
    elif kind == "worlds":
        n, joints = case["worlds"] * 125, case["worlds"] * 22
    else:
        n, joints = case["chains"] * (case["links"] + 1), case["chains"] * (3 * case["links"] + 1)
    contacts = n * CONTACTS[kind]
    passes = case.get("substeps", 4) * (1 + case.get("iterations", 8) + 4)
    # each body's descriptor, each contact's record and each joint's record in and out
    return {"bytes": n * 2 * 176 + contacts * 2 * 128 + joints * 2 * 304,
            "flops": passes * (contacts * 200 + joints * 250) + n * 13 * 300}


def exact(case, seed):
    """The learned warm start's gradients in 64 bits.  The other paths have no plain 64-bit
    form: a step is hundreds of sequential solver passes over contacts found by iterative
    overlap tests, whose discrete choices the rounding of the poses decides."""
    if case["kind"] != "mlp":
        return None
    X, T, p = _mlp_data(case, seed)
    X, T, p = X.astype(np.float64), T.astype(np.float64), p.astype(np.float64)
    n, at, part = len(X), 0, []
    h, i, o = abi.MLP_HID, abi.MLP_IN, abi.MLP_OUT
    for shape in ((h, i), (h,), (h, h), (h,), (o, h), (o,), (i,), (i,), (o,)):
        size = int(np.prod(shape))
        part.append(p[at:at + size].reshape(shape))
        at += size
    w1, b1, w2, b2, w3, b3, mean, scale, oscale = part
    x = (X - mean) * scale
    t = T / oscale
    z1 = x @ w1.T + b1
    a1 = np.maximum(z1, 0)
    z2 = a1 @ w2.T + b2
    a2 = np.maximum(z2, 0)
    d = a2 @ w3.T + b3 - t
    loss = (d ** 2).sum() / (3 * n)
    g = 2 * d / (3 * n)
    g2 = (g @ w3) * (z2 > 0)
    g1 = (g2 @ w2) * (z1 > 0)
    grads = [g1.T @ x, g1.sum(0), g2.T @ a1, g2.sum(0), g.T @ a2, g.sum(0)]
    return {"gradients": np.concatenate([v.ravel() for v in grads]), "loss": np.float64(loss)}
