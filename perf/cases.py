"""Performance cases: the work a program has this framework do, through its public entry points.

Each case is one call, or the few calls that belong together, of a real program:

  world    one world stepped and read back: a game's frame loop or an interactive scene. The bodies
           (circles, boxes and 3-8-gons, sizes 0.1-0.6 m) have settled in a walled container.
  pyramid  one world stepped and read back: the box pyramid on an edge ground, standing.
  gas      one world without gravity, every body in flight and colliding: the broadphase sees nearly
           all of its proxies move, as in a scene that is still falling.
  pile     one world of boxes settled into a deep pile: contacts and constraints, not motion.
  bridge   a world with revolute joints, a motor and limits and bodies lying on the planks, with
           sleeping allowed.
  rain     fast bodies and thin static plates with continuous physics (time of impact) on.
  batch    many independent worlds of uneven size stepped together: reinforcement learning and
           sampling; some steps per read-back.
  grad     one iteration of an optimisation through the physics: reset, taped steps, backward pass.
  queries  ray casts and box queries against a world: sensors, picking, line of sight.
  toi      stand-alone times of impact of pairs of moving shapes given as host arrays.

Worlds are brought to a state that lasts before a pass is run (settled, or in flight without loss of
energy), so that one pass costs what the next one does.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("box2d-rs_gb300"))
import b2g  # noqa: E402
import scenes  # noqa: E402

DT = 1.0 / 60.0
VI, PI = 8, 3  # velocity and position iterations of every configuration


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest world: what a step costs when there is nearly nothing to do
        {"name": "world_16", "kind": "world", "bodies": 16},
        # the 20-row pyramid of 210 boxes: the repository's smallest configuration
        {"name": "pyramid_210", "kind": "pyramid", "rows": 20},
        # a game level's worth of loose bodies, an odd number of them
        {"name": "world_3001", "kind": "world", "bodies": 3001},
        # 100k bodies of the mixed scene in flight: the flagship size
        {"name": "gas_100k", "kind": "gas", "bodies": 100_000},
        # 250k boxes in a pile: the largest single world
        {"name": "pile_250k", "kind": "pile", "bodies": 250_000},
        # the 30-plank bridge: the path of worlds with joints
        {"name": "bridge_30", "kind": "bridge", "planks": 30},
        # the path of continuous physics
        {"name": "rain_1000", "kind": "rain", "bodies": 1000},
        # 4096 worlds of 16 to 2048 bodies, 1.7 M bodies in all: the batched configuration
        {"name": "batch_4096", "kind": "batch", "worlds": 4096, "hi": 2048, "steps": 2},
        # the throw-and-stack gradient of one world, half of its 240 steps
        {"name": "grad_1", "kind": "grad", "worlds": 1, "steps": 120},
        # the same for 512 worlds at once
        {"name": "grad_512", "kind": "grad", "worlds": 512, "steps": 64},
        # a frame's rays and boxes against 20k bodies
        {"name": "queries_20k", "kind": "queries", "bodies": 20_000, "rays": 16_384, "boxes": 2048},
        # a large set of sweeps
        {"name": "toi_100k", "kind": "toi", "pairs": 100_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["world", "world", "pyramid", "gas", "pile", "bridge", "rain", "batch", "grad", "queries", "toi"])
    if kind == "world":
        return {"kind": kind, "bodies": _log(rng, 16, 60_000)}
    if kind == "pyramid":
        return {"kind": kind, "rows": rng.randint(5, 20)}
    if kind == "gas":
        return {"kind": kind, "bodies": _log(rng, 2000, 100_000)}
    if kind == "pile":
        return {"kind": kind, "bodies": _log(rng, 5000, 200_000)}
    if kind == "bridge":
        return {"kind": kind, "planks": rng.randint(10, 90)}
    if kind == "rain":
        return {"kind": kind, "bodies": _log(rng, 64, 4000)}
    if kind == "batch":
        return {"kind": kind, "worlds": _log(rng, 64, 2048), "hi": _log(rng, 64, 2048), "steps": rng.randint(1, 4)}
    if kind == "grad":
        return {"kind": kind, "worlds": _log(rng, 1, 256), "steps": rng.randint(20, 100)}
    if kind == "queries":
        return {"kind": kind, "bodies": _log(rng, 1000, 20_000), "rays": _log(rng, 256, 16_384), "boxes": _log(rng, 64, 2048)}
    return {"kind": kind, "pairs": _log(rng, 500, 100_000)}


# ---------------------------------------------------------------- scenes

def _mixed_fixtures(rng, first_body, n, friction=0.5, restitution=0.0):
    """n fixtures on bodies first_body...: a third each of circles, boxes and 3-8-gons."""
    f = b2g.fixture_defs(n)
    f["body"] = np.arange(first_body, first_body + n)
    f["density"] = 1.0
    f["friction"] = friction
    f["restitution"] = restitution
    kind = rng.integers(0, 3, n)
    size = rng.uniform(0.1, 0.6, n)
    c, b, g = kind == 0, kind == 1, kind == 2
    f["shape_type"] = np.where(c, b2g.CIRCLE, b2g.POLYGON)
    f["radius"][c] = 0.5 * size[c]
    f["polygon_mode"] = np.where(b, b2g.POLYGON_BOX, b2g.POLYGON_HULL)
    f["box_half_extents"][b] = (0.5 * size[b])[:, None] * rng.uniform(0.6, 1.0, (int(b.sum()), 2))
    # vertices at equal angles and radii that differ by at most a fifth: convex for 3 to 8 of them
    nv = rng.integers(3, 9, n)
    k = np.arange(8)
    angle = 2.0 * np.pi * k[None, :] / nv[:, None]
    radius = size[:, None] * rng.uniform(0.8, 1.0, (n, 8))
    v = np.stack([radius * np.cos(angle), radius * np.sin(angle)], 2)
    v[k[None, :] >= nv[:, None]] = 0.0
    f["vertices"][g] = v[g]
    f["vertex_count"][g] = nv[g]
    return f


def _container(width, height, lid=False, friction=0.5, restitution=0.0):
    """Fixtures of body 0: a floor, two walls and, with lid, a ceiling, as two-sided edges."""
    corners = [(0.0, height), (0.0, 0.0), (width, 0.0), (width, height), (0.0, height)][: 5 if lid else 4]
    f = b2g.fixture_defs(len(corners) - 1)
    f["shape_type"] = b2g.EDGE
    f["friction"] = friction
    f["restitution"] = restitution
    for i in range(len(corners) - 1):
        f["vertices"][i, 1], f["vertices"][i, 2] = corners[i], corners[i + 1]
    return f


def _grid_bodies(rng, n, cols, spacing, x0, y0):
    """n dynamic bodies on a jittered grid of that many columns, at random angles."""
    d = b2g.body_defs(n)
    d["allow_sleep"] = 0
    d["type"] = b2g.DYNAMIC
    i = np.arange(n)
    d["position"][:, 0] = x0 + (i % cols) * spacing + rng.uniform(-0.05, 0.05, n)
    d["position"][:, 1] = y0 + (i // cols) * spacing + rng.uniform(-0.05, 0.05, n)
    d["angle"] = rng.uniform(0.0, 2.0 * np.pi, n)
    return d


def _static_body():
    d = b2g.body_defs(1)
    d["type"] = b2g.STATIC
    return d


def _open(bodies, fixtures, gravity=(0.0, -10.0), num_worlds=1, joints=None, sleeping=False, continuous=False, settle=0,
          capacity=0):
    w = b2g.B2world(gravity=gravity, num_worlds=num_worlds, contact_capacity=capacity, pair_capacity=capacity)
    w.set_allow_sleeping(sleeping)
    w.set_continuous_physics(continuous)
    w.create_bodies(bodies)
    w.create_fixtures(fixtures)
    if joints is not None:
        w.create_joints(joints)
    for _ in range(settle):
        w.step(DT, VI, PI)
    w.synchronize()
    return w


def _prepare_world(case, rng):
    n = case["bodies"]
    rows = min(24, max(4, int(math.sqrt(n) / 2)))
    cols = -(-n // rows)
    bodies = np.concatenate([_static_body(), _grid_bodies(rng, n, cols, 1.3, 1.0, 1.0)])
    fixtures = np.concatenate([_container(cols * 1.3 + 0.7, 60.0), _mixed_fixtures(rng, 1, n)])
    return _open(bodies, fixtures, settle=200)


def _prepare_pyramid(case, rng):
    s = scenes.pyramid(rows=case["rows"])
    n = len(s["bodies"]) - 1
    s["bodies"]["position"][1:, 0] += rng.uniform(-0.01, 0.01, n).astype(np.float32)
    return _open(s["bodies"], s["fixtures"], settle=120)


def _prepare_gas(case, rng):
    n = case["bodies"]
    cols = int(math.ceil(math.sqrt(n)))
    d = _grid_bodies(rng, n, cols, 1.3, 1.0, 1.0)
    d["linear_velocity"] = rng.normal(0.0, 16.0, (n, 2))
    f = np.concatenate([_container(cols * 1.3 + 1.0, cols * 1.3 + 1.0, lid=True, friction=0.0, restitution=1.0),
                        _mixed_fixtures(rng, 1, n, friction=0.0, restitution=1.0)])
    f["restitution_threshold"] = 0.0  # no speed is too small to bounce: the gas keeps its energy
    return _open(np.concatenate([_static_body(), d]), f, gravity=(0.0, 0.0), settle=40)


def _prepare_pile(case, rng):
    n = case["bodies"]
    rows = 100
    cols = -(-n // rows)
    spacing = 0.43
    d = _grid_bodies(rng, n, cols, spacing, 0.3, 0.3)
    i = np.arange(n)
    d["position"][:, 0] = 0.3 + (i % cols) * spacing + rng.uniform(-0.005, 0.005, n)
    d["position"][:, 1] = 0.3 + (i // cols) * spacing
    d["angle"] = rng.uniform(-0.02, 0.02, n)
    f = b2g.fixture_defs(n)
    f["body"] = np.arange(1, n + 1)
    f["shape_type"] = b2g.POLYGON
    f["polygon_mode"] = b2g.POLYGON_BOX
    f["box_half_extents"] = rng.uniform(0.05, 0.2, (n, 2))
    f["density"] = 1.0
    f["friction"] = 0.6
    fixtures = np.concatenate([_container(cols * spacing + 0.3, 60.0, friction=0.6), f])
    # boxes this close together have many neighbours within their predicted boxes while they fall
    return _open(np.concatenate([_static_body(), d]), fixtures, settle=170, capacity=64 * n)


def _prepare_bridge(case, rng):
    planks = case["planks"]
    s = scenes.bridge(planks=planks, seed=int(rng.integers(1 << 30)), drops=planks)
    return _open(s["bodies"], s["fixtures"], joints=s["joints"], sleeping=True, settle=240)


def _prepare_rain(case, rng):
    """Bodies at 20-90 m/s between thin plates in a closed box, without gravity or loss."""
    n = case["bodies"]
    cols = int(math.ceil(math.sqrt(2.0 * n)))
    rows = -(-n // cols)
    side_x, side_y = cols * 3.0 + 4.0, rows * 3.0 + 4.0
    plates = b2g.body_defs(cols // 3 + 1)
    plates["type"] = b2g.STATIC
    plates["position"][:, 0] = 3.5 + np.arange(len(plates)) * 9.0
    plates["position"][:, 1] = rng.uniform(0.2, 0.8, len(plates)) * side_y
    pf = b2g.fixture_defs(len(plates))
    pf["body"] = np.arange(1, len(plates) + 1)
    pf["shape_type"] = b2g.POLYGON
    pf["polygon_mode"] = b2g.POLYGON_BOX
    pf["box_half_extents"] = (3.0, 0.05)
    pf["friction"] = 0.0
    pf["restitution"] = 1.0
    first = 1 + len(plates)
    d = _grid_bodies(rng, n, cols, 3.0, 3.0, 3.0)
    speed, heading = rng.uniform(20.0, 90.0, n), rng.uniform(0.0, 2.0 * np.pi, n)
    d["linear_velocity"] = np.stack([speed * np.cos(heading), speed * np.sin(heading)], 1)
    f = np.concatenate([_container(side_x, side_y, lid=True, friction=0.0, restitution=1.0), pf,
                        _mixed_fixtures(rng, first, n, friction=0.0, restitution=1.0)])
    f["restitution_threshold"] = 0.0
    return _open(np.concatenate([_static_body(), plates, d]), f, gravity=(0.0, 0.0), continuous=True, settle=20)


def _batch_counts(case):
    """Bodies of each world: log-uniform from 16 to hi, as spread over the quantiles."""
    u = (np.arange(case["worlds"]) + 0.5) / case["worlds"]
    return np.exp(math.log(16.0) + u * (math.log(case["hi"]) - math.log(16.0))).astype(np.int64)


def _prepare_batch(case, rng):
    counts = rng.permutation(_batch_counts(case))
    nw, total = len(counts), int(counts.sum())
    spacing = 1.3
    cols = np.ceil(2.0 * np.sqrt(counts)).astype(np.int64)
    # world by world: its ground, then its bodies on a grid
    world = np.repeat(np.arange(nw), counts + 1)
    start = np.concatenate([[0], np.cumsum(counts + 1)[:-1]])
    place = np.arange(total + nw) - start[world] - 1
    ground = place < 0
    bodies = b2g.body_defs(total + nw)
    bodies["allow_sleep"] = 0
    bodies["world_index"] = world
    bodies["type"] = np.where(ground, b2g.STATIC, b2g.DYNAMIC)
    c, m = cols[world], total + nw
    bodies["position"][:, 0] = np.where(ground, 0.0, (place % c - 0.5 * c) * spacing + rng.uniform(-0.05, 0.05, m))
    bodies["position"][:, 1] = np.where(ground, 0.0, 1.0 + (place // c) * spacing + rng.uniform(-0.05, 0.05, m))
    bodies["angle"] = np.where(ground, 0.0, rng.uniform(0.0, 2.0 * np.pi, m))
    f = _mixed_fixtures(rng, 0, m)
    half = 0.5 * cols * spacing + 5.0
    e = np.zeros((nw, 8, 2), np.float32)
    e[:, 1, 0], e[:, 2, 0] = -half, half
    f["shape_type"][ground] = b2g.EDGE
    f["radius"][ground] = b2g.fixture_defs(1)["radius"][0]
    f["vertices"][ground] = e
    f["density"][ground] = 0.0
    return _open(bodies, f, num_worlds=nw, settle=120)


def _prepare_grad(case, rng):
    nw = case["worlds"]
    s = scenes.throw_stack()
    nb = len(s["bodies"])
    bodies, fixtures = np.tile(s["bodies"], nw), np.tile(s["fixtures"], nw)
    bodies["world_index"] = np.repeat(np.arange(nw), nb)
    fixtures["body"] += np.repeat(np.arange(nw) * nb, len(s["fixtures"])).astype(np.uint32)
    thrown = s["projectile"] + np.arange(nw) * nb
    bodies["linear_velocity"][thrown] = np.stack([rng.uniform(10.0, 14.0, nw), rng.uniform(2.0, 4.0, nw)], 1)
    w = _open(bodies, fixtures, num_worlds=nw)
    # the projectile has just met the stack when the taped steps begin
    for _ in range(30):
        w.step(DT, VI, PI)
    return {"world": w, "initial": w.save_state(), "steps": case["steps"],
            "stack": s["stack"][None, :] + (np.arange(nw) * nb)[:, None],
            "target": np.array([6.0, 1.0]) + rng.uniform(0.0, 1.0, (nw, 2)),
            "out": np.zeros(nw * nb, b2g.BODY_STATE), "slots": case["steps"] * nw * 320}


def _query_scene(case, seed):
    """(bodies, fixtures, rays, boxes): bodies at rest in space and what is asked of them."""
    rng = np.random.default_rng(seed)
    n = case["bodies"]
    cols = int(math.ceil(math.sqrt(n)))
    bodies = _grid_bodies(rng, n, cols, 1.3, 0.0, 0.0)
    fixtures = _mixed_fixtures(rng, 0, n)
    side, nr, nq = cols * 1.3, case["rays"], case["boxes"]
    p = rng.uniform(0.0, side, (nr, 2))
    length, heading = rng.uniform(3.0, 30.0, nr), rng.uniform(0.0, 2.0 * np.pi, nr)
    rays = np.concatenate([p, p + np.stack([length * np.cos(heading), length * np.sin(heading)], 1)], 1)
    lo = rng.uniform(0.0, side, (nq, 2))
    boxes = np.concatenate([lo, lo + rng.uniform(0.5, 6.0, (nq, 2))], 1)
    return bodies, fixtures, rays.astype(np.float32), boxes.astype(np.float32)


def _toi_scene(case, rng):
    """Pairs of circles, 3-8-gons and edges that move up to 4 m and turn up to 3 rad."""
    n = case["pairs"]

    def defs():
        d = b2g.fixture_defs(n)
        kind = rng.integers(0, 3, n)
        c, p, e = kind == 0, kind == 1, kind == 2
        d["shape_type"][c] = b2g.CIRCLE
        d["radius"][c] = rng.uniform(0.1, 0.6, int(c.sum()))
        d["vertices"][c, 0] = rng.uniform(-0.2, 0.2, (int(c.sum()), 2))
        d["shape_type"][p] = b2g.POLYGON
        d["polygon_mode"][p] = b2g.POLYGON_HULL
        k = rng.integers(3, 9, n)
        ang = np.sort(rng.uniform(0.0, 2.0 * np.pi, (n, 8)), axis=1)
        rad = rng.uniform(0.2, 0.7, (n, 8))
        v = np.stack([rad * np.cos(ang), rad * np.sin(ang)], 2).astype(np.float32)
        v[np.arange(8)[None, :] >= k[:, None]] = 0.0
        d["vertices"][p] = v[p]
        d["vertex_count"][p] = k[p]
        d["shape_type"][e] = b2g.EDGE
        a = rng.uniform(-2.0, 2.0, (n, 2)).astype(np.float32)
        d["vertices"][e, 1] = a[e]
        d["vertices"][e, 2] = (a + rng.uniform(-3.0, 3.0, (n, 2)))[e]
        return d

    def sweeps(spread):
        s = np.zeros(n, b2g.SWEEP)
        s["local_center"] = rng.uniform(-0.1, 0.1, (n, 2))
        s["c0"] = rng.uniform(-spread, spread, (n, 2))
        s["c"] = s["c0"] + rng.uniform(-spread, spread, (n, 2))
        s["a0"] = rng.uniform(-10.0, 10.0, n)
        s["a"] = s["a0"] + rng.uniform(-3.0, 3.0, n)
        return s

    return defs(), sweeps(4.0), defs(), sweeps(1.0)


_WORLDS = {"world": _prepare_world, "pyramid": _prepare_pyramid, "gas": _prepare_gas, "pile": _prepare_pile,
           "bridge": _prepare_bridge, "rain": _prepare_rain, "batch": _prepare_batch}


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in _WORLDS:
        w = _WORLDS[kind](case, rng)
        return {"kind": "step", "world": w, "steps": case.get("steps", 1), "out": np.zeros(w.body_count, b2g.BODY_STATE)}
    if kind == "grad":
        return {"kind": kind, **_prepare_grad(case, rng)}
    if kind == "queries":
        bodies, fixtures, rays, boxes = _query_scene(case, seed)
        w = _open(bodies, fixtures, gravity=(0.0, 0.0), settle=1)
        # the program keeps what its boxes found in a table of its own, -1 past the end
        return {"kind": kind, "world": w, "rays": rays, "boxes": boxes, "found": np.full((24 * len(boxes), 2), -1, np.int32)}
    return {"kind": kind, "pairs": _toi_scene(case, rng)}


# ---------------------------------------------------------------- one pass

def _floats(states):
    """Body states as the eight numbers of each body."""
    return states.view(np.float32).reshape(-1, 8)


def run(state):
    kind = state["kind"]
    if kind == "step":
        w = state["world"]
        for _ in range(state["steps"]):
            w.step(DT, VI, PI)
        return _floats(w.get_body_states(out=state["out"]))
    if kind == "grad":
        w = state["world"]
        w.load_state(state["initial"])
        w.tape_begin(state["steps"], 16, state["slots"])
        for _ in range(state["steps"]):
            w.step(DT, VI, PI)
        w.tape_end()
        final = w.get_body_states(out=state["out"])
        # the loss: each stack's centre of mass to its target, squared
        off = final["world_center"][state["stack"]].astype(np.float64).mean(1) - state["target"]
        d = np.zeros(len(final), b2g.BODY_STATE)
        d["world_center"][state["stack"]] = (2.0 * off / state["stack"].shape[1])[:, None, :]
        return {"final": _floats(final), "gradient": _floats(w.backward(d))}
    if kind == "queries":
        hits = state["world"].ray_cast_closest(state["rays"])
        pairs = state["world"].query_aabb(state["boxes"])
        found = state["found"]
        found[: len(pairs)] = pairs
        found[len(pairs):] = -1
        return {"fixture": hits["fixture"], "fraction": hits["fraction"], "normal": hits["normal"],
                "point": hits["point"], "pairs": found}
    da, sa, db, sb = state["pairs"]
    hits = b2g.time_of_impact(da, sa, db, sb)
    return {"state": hits["state"], "t": hits["t"]}


# ---------------------------------------------------------------- what a pass cannot do without

# A body's state is read and written once a step (position, angle, velocities: 24 B each way) and its
# shape read once (about 80 B); a live contact's record (its manifold, impulses and ids, 80 B) is read
# and written once. A constraint takes about 140 operations in each velocity iteration and 120 in each
# position iteration; a body about 60 for its integration and its box.
def _step_work(bodies, contacts, constraints):
    return {"bytes": bodies * (48 + 80) + contacts * 160,
            "flops": bodies * 60 + contacts * 100 + constraints * (VI * 140 + PI * 120)}


def work(case):
    kind = case["kind"]
    if kind in ("grad", "batch", "pile", "world", "pyramid", "gas", "bridge", "rain"):
        n = {"grad": lambda: 65 * case["worlds"], "batch": lambda: int(_batch_counts(case).sum()),
             "pyramid": lambda: case["rows"] * (case["rows"] + 1) // 2,
             "bridge": lambda: 2 * case["planks"]}.get(kind, lambda: case["bodies"])()
        # contacts and constraints for each body: counted once, rounded
        contacts, constraints = {"world": (5.4, 2.0), "batch": (4.6, 1.8), "pile": (9.2, 2.6), "gas": (2.8, 0.1),
                                 "rain": (1.8, 0.03), "bridge": (1.4, 1.0), "pyramid": (2.8, 1.9), "grad": (3.4, 1.3)}[kind]
        step = _step_work(n, n * contacts, n * constraints)
        out = n * 32
        if kind == "grad":  # the forward steps, then as many of the replay and of the adjoint
            return {"bytes": case["steps"] * (step["bytes"] + n * constraints * 144 * 2) + 3 * out,
                    "flops": case["steps"] * 4 * step["flops"]}
        k = case.get("steps", 1)
        return {"bytes": k * step["bytes"] + out, "flops": k * step["flops"]}
    if kind == "queries":  # the bodies once; each ray meets the shapes along it, each box those in it
        return {"bytes": case["bodies"] * 96 + case["rays"] * (16 + 24) + case["boxes"] * (16 + 8 * 8),
                "flops": case["rays"] * 10 * 60 + case["boxes"] * 8 * 4}
    pair = b2g.FIXTURE_DEF.itemsize * 2 + b2g.SWEEP.itemsize * 2 + b2g.TOI_OUTPUT.itemsize
    return {"bytes": case["pairs"] * pair, "flops": case["pairs"] * 3000}


# ---------------------------------------------------------------- what the outputs are in 64 bits

def _ray_hits(case, seed):
    """Closest hit of each ray in 64 bits: every ray against every body whose box its own box meets."""
    bodies, fixtures, rays, _ = _query_scene(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def t(a):
        return torch.from_numpy(np.ascontiguousarray(a, np.float64)).to(dev)

    n = len(bodies)
    pos, angle = t(bodies["position"]), t(bodies["angle"])
    circle = torch.from_numpy(fixtures["shape_type"] == b2g.CIRCLE).to(dev)
    box = fixtures["polygon_mode"] == b2g.POLYGON_BOX
    local = fixtures["vertices"].astype(np.float64)
    count = fixtures["vertex_count"].astype(np.int64)
    h = fixtures["box_half_extents"].astype(np.float64)
    local[box] = 0.0
    local[box, :4] = (np.array([[-1, -1], [1, -1], [1, 1], [-1, 1]])[None] * h[:, None, :])[box]
    count[box] = 4
    count = torch.from_numpy(count).to(dev)
    radius = t(fixtures["radius"])
    local = t(local)
    # polygons in the world: vertices and outward normals of their edges
    c, s = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
    v = torch.stack([c * local[..., 0] - s * local[..., 1], s * local[..., 0] + c * local[..., 1]], 2) + pos[:, None, :]
    k = torch.arange(8, device=dev)[None, :]
    nxt = torch.where(k + 1 < count[:, None], k + 1, torch.zeros_like(k))
    edge = torch.gather(v, 1, nxt[..., None].expand(n, 8, 2)) - v
    normal = torch.stack([edge[..., 1], -edge[..., 0]], 2)
    normal = normal / normal.norm(dim=2, keepdim=True).clamp_min(1e-30)
    used = k < count[:, None]
    reach = torch.where(circle, radius, torch.where(used, (v - pos[:, None, :]).norm(dim=2), torch.zeros_like(v[..., 0])).amax(1))
    p1, p2 = t(rays[:, :2]), t(rays[:, 2:])
    lo, hi = torch.minimum(p1, p2), torch.maximum(p1, p2)
    best = torch.full((len(rays),), math.inf, dtype=torch.float64, device=dev)
    best_n = torch.zeros((len(rays), 2), dtype=torch.float64, device=dev)
    for at in range(0, len(rays), 512):
        a, b = lo[at:at + 512], hi[at:at + 512]
        near = ((pos[None] + reach[None, :, None] >= a[:, None]) & (pos[None] - reach[None, :, None] <= b[:, None])).all(2)
        r, f = near.nonzero(as_tuple=True)
        r = r + at
        o, d = p1[r], p2[r] - p1[r]
        # circles
        m = o - pos[f]
        rr, md = (d * d).sum(1), (m * d).sum(1)
        sigma = md * md - rr * ((m * m).sum(1) - radius[f] ** 2)
        tc = -(md + sigma.clamp_min(0.0).sqrt()) / rr
        hit_c = (sigma >= 0) & (tc >= 0) & (tc <= 1)
        nc = m + tc[:, None] * d
        nc = nc / nc.norm(dim=1, keepdim=True).clamp_min(1e-30)
        # polygons: the last entering edge, not before 0.032 of the ray, ahead of the first leaving one
        num = (normal[f] * (v[f] - o[:, None, :])).sum(2)
        den = (normal[f] * d[:, None, :]).sum(2)
        ok = used[f]
        tt = num / torch.where(den == 0, torch.ones_like(den), den)
        enter = torch.where(ok & (den < 0), tt, torch.full_like(tt, -math.inf))
        leave = torch.where(ok & (den > 0), tt, torch.full_like(tt, math.inf)).amin(1)
        outside = (ok & (den == 0) & (num < 0)).any(1)
        tp, ip = enter.max(1)
        start = float(np.float32(0.032))
        hit_p = (tp > start) & (tp <= 1) & (leave >= tp) & ~outside
        npoly = normal[f, ip]
        is_c = circle[f]
        hit = torch.where(is_c, hit_c, hit_p)
        tm = torch.where(hit, torch.where(is_c, tc, tp), torch.full_like(tc, math.inf))
        nn = torch.where(is_c[:, None], nc, npoly)
        best.scatter_reduce_(0, r, tm, "amin")
        first = hit & (tm == best[r])
        best_n[r[first]] = nn[first]
    none = torch.isinf(best)
    frac = torch.where(none, torch.ones_like(best), best)
    point = (1.0 - frac)[:, None] * p1 + frac[:, None] * p2
    point[none] = 0.0
    return frac, best_n, point


def exact(case, seed):
    """Rays have a value that plain arithmetic gives. A step's outputs depend on the order in which its
    constraints are solved, and a time of impact on where its iteration stops: those have none."""
    if case["kind"] != "queries":
        return None
    frac, normal, point = _ray_hits(case, seed)
    return {"fixture": None, "fraction": frac, "normal": normal, "point": point, "pairs": None}
