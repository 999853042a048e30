"""The measured work: what a program that uses this library has it do, through its public entry points.

Kinds of case:

- rollout: one world or a batch of worlds is put back to a saved state and advanced some steps, then every body's pose,
  velocity and state is read (an episode of a learning environment, a what-if from a saved game or robot state). The
  state is a checkpoint taken `settle` steps after the bodies were dropped, so that contacts, warm starts and sleeping
  islands are there as in a running simulation.
- flight: the same call over bodies that touch nothing yet (debris, projectiles, the first frames of a scene).
- collide: one collision-detection pass over a world (poses, boxes, tree, pairs, contact manifolds) and its manifolds.
- serve: requests of different sizes handed to the request server at once, and their results.
- query: box and circle queries against a settled pile (picking, area effects, sensors).
- joints: motor-driven chains of revolute joints with springs between neighbouring links, advanced some steps.
"""
import math
import os
import sys

import numpy as np

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "physicssimulation-agony_b200"))
import ag2d  # noqa: E402
from ag2d import scenes  # noqa: E402

DT = 1.0 / 60.0
GRAVITY = -9.81


def listed():
    return [
        # One small world, a few dozen bodies: an interactive scene or a single environment. Launches and latency.
        dict(name="world_64", kind="rollout", scene="drop", worlds=1, bodies=64, settle=60, steps=16, iterations=8,
             ccd=False),
        # The plain single world of the benchmark's first configuration, with its pile on the ground.
        dict(name="world_2048", kind="rollout", scene="drop", worlds=1, bodies=2048, settle=300, steps=16, iterations=8,
             ccd=False),
        # The large single world: boxes, circles and polygons piling up in a container.
        dict(name="pile_100k", kind="rollout", scene="container", worlds=1, bodies=100_000, settle=300, steps=8,
             iterations=8, ccd=False),
        # A vector of small equal environments with every shape, capsules among them, odd sizes.
        dict(name="envs_64x61", kind="rollout", scene="capsules", worlds=64, bodies=61, settle=60, steps=16,
             iterations=8, ccd=False),
        # A ragged batch of middling worlds with small fast bodies, continuous collision on.
        dict(name="ragged_509_ccd", kind="rollout", scene="fast", worlds=509, bodies=1536, settle=90, steps=16,
             iterations=8, ccd=True),
        # The batched benchmark: 4,096 worlds of 16 to 2,048 bodies in their settled window.
        dict(name="batch_4096", kind="rollout", scene="drop", worlds=4096, bodies=2048, settle=300, steps=20,
             iterations=8, ccd=False),
        # Bodies in free flight, nothing touching yet.
        dict(name="flight_20k", kind="flight", bodies=20_000, steps=12),
        # Collision detection alone, an odd middling size and the benchmark's million bodies.
        dict(name="collide_20011", kind="collide", bodies=20_011),
        dict(name="collide_1m", kind="collide", bodies=1_000_000),
        # A burst of requests at the server, log-uniform sizes, continuous collision on.
        dict(name="serve_48", kind="serve", requests=48, bodies=2048, steps=40),
        # Sixteen queries on a settled pile.
        dict(name="query_20k", kind="query", bodies=20_000, settle=240, queries=16),
        # Jointed machines: 960 links on chains of twelve, motors on every fourth link.
        dict(name="joints_960", kind="joints", bodies=960, steps=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["world", "batch", "batch", "collide", "flight", "serve", "query", "joints"])
    if kind == "world":
        scene = rng.choice(["drop", "container", "capsules", "fast"])
        return dict(kind="rollout", scene=scene, worlds=1,
                    bodies=_log_int(rng, 24, 8000 if scene in ("drop", "fast") else 60_000),
                    settle=rng.randint(40, 300), steps=rng.randint(6, 20), iterations=rng.choice([4, 8, 8, 12]),
                    ccd=scene == "fast")
    if kind == "batch":
        worlds = _log_int(rng, 8, 2500)
        scene = rng.choice(["drop", "drop", "capsules", "fast"])
        return dict(kind="rollout", scene=scene, worlds=worlds,
                    bodies=_log_int(rng, 24, min(2048, 600_000 // worlds)), settle=rng.randint(40, 240),
                    steps=rng.randint(6, 20), iterations=rng.choice([4, 8, 8]), ccd=scene == "fast")
    if kind == "collide":
        return dict(kind="collide", bodies=_log_int(rng, 3000, 900_000))
    if kind == "flight":
        return dict(kind="flight", bodies=_log_int(rng, 100, 60_000), steps=rng.randint(4, 16))
    if kind == "serve":
        return dict(kind="serve", requests=rng.randint(6, 60), bodies=_log_int(rng, 128, 2048),
                    steps=rng.randint(16, 48))
    if kind == "query":
        return dict(kind="query", bodies=_log_int(rng, 500, 40_000), settle=rng.randint(60, 240),
                    queries=rng.randint(4, 24))
    return dict(kind="joints", bodies=12 * _log_int(rng, 4, 160), steps=rng.randint(6, 20))


# ---------------------------------------------------------------------------------------------------------------
# Scenes: the shapes, sizes and distributions of ag2d.scenes, built without a Python loop over the bodies.
# ---------------------------------------------------------------------------------------------------------------
def _polygons(rng, radius, lo=3, hi=8):
    """Convex outlines on circles of these radii, each radius jittered by 15 %: (counts, offsets, xy, areas)."""
    n = radius.size
    counts = rng.integers(lo, hi + 1, n).astype(np.int32)
    offsets = np.zeros(n, np.int64)
    if n:
        offsets[1:] = np.cumsum(counts[:-1])
    total = int(counts.sum())
    owner = np.repeat(np.arange(n), counts)
    k = np.arange(total) - offsets[owner]
    phase = rng.uniform(0.0, 1.0, n) * 2.0 * math.pi / np.maximum(counts, 1)
    ang = phase[owner] + 2.0 * math.pi * k / counts[owner]
    r = radius[owner] * rng.uniform(0.85, 1.15, total)
    xy = np.stack([r * np.cos(ang), r * np.sin(ang)], axis=1).astype(np.float32)
    nxt = np.where(k + 1 < counts[owner], np.arange(total) + 1, offsets[owner])
    x, y = xy[:, 0].astype(np.float64), xy[:, 1].astype(np.float64)
    area = np.zeros(n)
    np.add.at(area, owner, 0.5 * (x * y[nxt] - x[nxt] * y))
    return counts, offsets, xy, area


def _scene(name, static_boxes, kind, x, y, radius=None, width=None, height=None, rot=None, vel=None, spin=None,
           polygons=None, gravity=(0.0, GRAVITY), iterations=8):
    """Static boxes (x, y, width, height) first, then the given bodies, density 1."""
    ns, n = len(static_boxes), kind.size
    f = lambda a: np.zeros(n, np.float32) if a is None else np.asarray(a, np.float32)
    radius, width, height, rot, spin = f(radius), f(width), f(height), f(rot), f(spin)
    vel = np.zeros((n, 2), np.float32) if vel is None else np.asarray(vel, np.float32)
    poly = kind == scenes.POLYGON
    counts, offsets = np.zeros(n, np.int32), np.zeros(n, np.int64)
    xy, area = np.zeros((0, 2), np.float32), np.zeros(n)
    if polygons is not None:
        counts[poly], offsets[poly], xy, area[poly] = polygons
    mass = np.select([kind == scenes.CIRCLE, kind == scenes.BOX, kind == scenes.CAPSULE],
                     [math.pi * radius * radius, width * height, 2.0 * width * radius + math.pi * radius * radius], area)
    st = np.asarray(static_boxes, np.float32).reshape(ns, 4)
    z = np.zeros(ns, np.float32)
    cat = lambda a, b: np.concatenate([a, b.astype(a.dtype)])
    return scenes.Scene(
        kind=cat(np.full(ns, scenes.BOX, np.uint8), kind), px=cat(st[:, 0], x), py=cat(st[:, 1], y), rot=cat(z, rot),
        vx=cat(z, vel[:, 0]), vy=cat(z, vel[:, 1]), w=cat(z, spin), mass=cat(z, mass), radius=cat(z, radius),
        width=cat(st[:, 2], width), height=cat(st[:, 3], height), poly_offset=cat(np.zeros(ns, np.int64), offsets),
        poly_count=cat(np.zeros(ns, np.int32), counts), poly_xy=xy, material=np.ones(ns + n, np.uint32),
        materials=[scenes.FRICTION_MATERIAL], dt=DT, velocity_iterations=iterations, gravity=gravity, name=name)


def _drop(rng, n, fast=False, iterations=8):
    """Polygons of 3 to 8 vertices above a ground box, the density of 2,048 bodies in 200 x 100 m; with `fast`, one
    in twenty is a small circle at 200 m/s instead."""
    scale = math.sqrt(n / 2048.0)
    w, h = max(20.0, 200.0 * scale), max(10.0, 100.0 * scale)
    x, y = rng.uniform(-0.5 * w, 0.5 * w, n), rng.uniform(2.5, 2.5 + h, n)
    kind = np.full(n, scenes.POLYGON, np.uint8)
    vel, radius = np.zeros((n, 2)), np.zeros(n)
    if fast:
        small = rng.random(n) < 0.05
        kind[small], radius[small] = scenes.CIRCLE, 0.05
        ang = rng.uniform(-0.75 * math.pi, -0.25 * math.pi, n)
        vel[small] = 200.0 * np.stack([np.cos(ang), np.sin(ang)], axis=1)[small]
    polys = _polygons(rng, rng.uniform(0.5, 2.0, int((kind == scenes.POLYGON).sum())))
    return _scene("drop", [(0.0, -1.0, 220.0, 2.0)], kind, x, y, radius=radius, vel=vel, polygons=polys,
                  iterations=iterations)


def _container(rng, n, capsules=False, iterations=8):
    """Mixed bodies, one per cell of a grid forty rows high (or square, when small) above the floor of a container."""
    cell = 4.8
    columns = max(n // 40, int(math.ceil(math.sqrt(n))) if n < 1600 else 1)
    rows = (n + columns - 1) // columns
    inner, wall = columns * cell, rows * cell + 20.0
    boxes = [(0.0, -1.0, inner + 4.0, 2.0), (-0.5 * inner - 1.0, 0.5 * wall, 2.0, wall),
             (0.5 * inner + 1.0, 0.5 * wall, 2.0, wall)]
    i = np.arange(n)
    x = -0.5 * inner + (i % columns + 0.5) * cell
    y = 0.5 * cell + (i // columns) * cell
    u = rng.random(n)
    if capsules:
        kind = np.select([u < 0.30, u < 0.55, u < 0.75], [scenes.CAPSULE, scenes.BOX, scenes.CIRCLE], scenes.POLYGON)
    else:
        kind = np.select([u < 0.60, u < 0.85], [scenes.BOX, scenes.CIRCLE], scenes.POLYGON)
    kind = kind.astype(np.uint8)
    cap, box = kind == scenes.CAPSULE, kind == scenes.BOX
    side = rng.uniform(0.3, 1.5, n)
    width = np.where(cap, rng.uniform(0.4, 2.4, n), np.where(box, side, 0.0))
    height = np.where(box, side, 0.0)
    radius = np.where(cap, rng.uniform(0.15, 0.6, n), np.where(kind == scenes.CIRCLE, rng.uniform(0.2, 1.0, n), 0.0))
    rot = np.where(cap, rng.uniform(0.0, math.pi, n), 0.0)
    polys = _polygons(rng, rng.uniform(0.5, 2.0, int((kind == scenes.POLYGON).sum())))
    return _scene("container", boxes, kind, x, y, radius=radius, width=width, height=height, rot=rot, polygons=polys,
                  iterations=iterations)


def _gas(rng, n):
    """Circles and 4 to 6-gons of log-uniform size in a square, no gravity: the density of a million in 4 x 4 km."""
    extent = 4.0 * math.sqrt(n)
    size = np.exp(rng.uniform(math.log(0.1), math.log(2.0), n))
    kind = np.where(rng.random(n) < 0.5, scenes.CIRCLE, scenes.POLYGON).astype(np.uint8)
    x, y = rng.uniform(-0.5 * extent, 0.5 * extent, n), rng.uniform(-0.5 * extent, 0.5 * extent, n)
    polys = _polygons(rng, size[kind == scenes.POLYGON], 4, 6)
    return _scene("gas", [], kind, x, y, radius=np.where(kind == scenes.CIRCLE, size, 0.0),
                  vel=rng.normal(0.0, 5.0, (n, 2)), polygons=polys, gravity=(0.0, 0.0))


def _flight(case, seed):
    """Boxes and circles on a wide grid high above the ground, thrown and spinning."""
    rng = np.random.default_rng(seed)
    n = case["bodies"]
    columns = int(math.ceil(math.sqrt(n)))
    i = np.arange(n)
    x, y = (i % columns - 0.5 * columns) * 6.0, 200.0 + (i // columns) * 6.0
    kind = np.where(rng.random(n) < 0.6, scenes.BOX, scenes.CIRCLE).astype(np.uint8)
    side = np.where(kind == scenes.BOX, rng.uniform(0.3, 1.5, n), 0.0)
    return _scene("flight", [(0.0, -1.0, 220.0, 2.0)], kind, x, y, radius=np.where(
        kind == scenes.CIRCLE, rng.uniform(0.2, 1.0, n), 0.0), width=side, height=side,
        vel=rng.uniform(-2.0, 2.0, (n, 2)), spin=rng.uniform(0.5, 3.0, n))


def _one_scene(rng, scene, n, iterations):
    if scene == "container":
        return _container(rng, n, iterations=iterations)
    if scene == "capsules":
        return _container(rng, n, capsules=True, iterations=iterations)
    return _drop(rng, n, fast=scene == "fast", iterations=iterations)


def _counts(case):
    """Body counts of the worlds: log-uniform from 16 (requests: 32) for the ragged scenes, all alike for the capsule
    environments. They belong to the case: its seeds differ in shapes and places."""
    rng = np.random.default_rng(case["bodies"])
    if case["kind"] == "serve":
        return scenes.log_uniform_counts(rng, case["requests"], 32, case["bodies"])
    if case["worlds"] == 1 or case["scene"] == "capsules":
        return np.full(case["worlds"], case["bodies"], np.int64)
    return scenes.log_uniform_counts(rng, case["worlds"], 16, case["bodies"])


# ---------------------------------------------------------------------------------------------------------------
# What a program holds before the call, and the call.
# ---------------------------------------------------------------------------------------------------------------
def _outputs(engine):
    """Page-locked destinations for what a rollout reads."""
    nb, _ = engine.counts()
    return {"pose": ag2d.host_empty(12 * nb), "vx": ag2d.host_empty(4 * nb), "vy": ag2d.host_empty(4 * nb),
            "spin": ag2d.host_empty(4 * nb), "state": ag2d.host_empty(4 * nb)}


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind in ("rollout", "flight"):
        if kind == "flight":
            worlds = [ag2d.World.from_scene(_flight(case, seed))]
        else:
            worlds = [ag2d.World.from_scene(_one_scene(rng, case["scene"], int(n), case["iterations"]), ccd=case["ccd"])
                      for n in _counts(case)]
        batch = ag2d.Batch(worlds)
        for w in worlds:
            w.close()
        batch.step(case.get("settle", 0))
        return {"case": case, "batch": batch, "start": batch.save(), "out": _outputs(batch.engine)}
    if kind == "collide":
        w = ag2d.World.from_scene(_gas(rng, case["bodies"]))
        # The program knows how many contacts its scene has at most and keeps page-locked room for them.
        room = int(0.25 * case["bodies"]) + 1024
        out = ag2d.host_empty(room * ag2d.MANIFOLD_DTYPE.itemsize)
        out[:] = 0
        return {"case": case, "world": w, "out": out}
    if kind == "serve":
        counts = _counts(case)
        worlds = [ag2d.World.from_scene(_drop(rng, int(n), fast=True), ccd=True) for n in counts]
        server = ag2d.Server(memory_budget_bytes=8 << 30, steps_per_round=8, ccd=True, reserve_bodies=int(counts.sum()))
        return {"case": case, "server": server, "worlds": worlds}
    if kind == "query":
        w = ag2d.World.from_scene(_container(rng, case["bodies"]))
        w.step(case["settle"])
        x, y = w.read(ag2d.BODY_COM_X), w.read(ag2d.BODY_COM_Y)
        at = rng.integers(3, x.size, case["queries"])   # around bodies of the pile
        half = rng.uniform(0.5, 12.0, case["queries"])
        room = 1200 * case["queries"]
        return {"case": case, "world": w, "at": [(float(x[i]), float(y[i]), float(h)) for i, h in zip(at, half)],
                "found": np.zeros(room, np.uint32), "touched": np.zeros(room, np.uint32),
                "distance": np.zeros(room, np.float32)}
    # joints: chains of twelve links hanging from one anchor each, motors on every fourth link, springs between the
    # links of neighbouring chains.
    w = ag2d.World(sleep_time=1.0e6)
    mat = w.add_material(*scenes.FRICTION_MATERIAL)
    before = None
    for c in range(case["bodies"] // 12):
        x0 = 30.0 * c
        prev = w.create_body(x0, 50.0, mass=0.0, inertia=0.0)
        links = []
        for k in range(12):
            b = w.create_body(x0 + 1.0 + k, 50.0, mass=1.0 + 0.1 * k, inertia=0.1 + 0.1 * float(rng.random()))
            w.add_collider(b, scenes.CIRCLE, radius=0.2, material=mat)
            w.create_revolute_joint(prev, b, (0.5, 0.0) if k else (0.0, 0.0), (-0.5, 0.0), 5.0e4, 50.0)
            if k % 4 == 0:
                w.create_motor(b, float(rng.uniform(-2.0, 2.0)), float(rng.uniform(5.0, 9.0)))
            links.append(b)
            prev = b
        if before is not None:
            for k in range(2, 12, 3):
                w.create_spring(before[k], links[k], (0.0, 0.0), (0.0, 0.0), 28.0, 40.0, 2.0)
        before = links
    w.step(1)
    return {"case": case, "world": w, "out": _outputs(w)}


def _read_bodies(engine, out):
    return {"pose": engine.read(ag2d.BODY_POSE, out["pose"]), "vx": engine.read(ag2d.BODY_VEL_X, out["vx"]),
            "vy": engine.read(ag2d.BODY_VEL_Y, out["vy"]),
            "spin": engine.read(ag2d.BODY_ANGULAR_VELOCITY, out["spin"]),
            "state": engine.read(ag2d.BODY_STATE, out["state"])}


def _gather(parts, room):
    """The parts one after the other at the front of `room`."""
    n = sum(p.size for p in parts)
    np.concatenate(parts, out=room[:n])
    return room


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("rollout", "flight"):
        batch = state["batch"]
        batch.load(state["start"])
        batch.step(case["steps"])
        return _read_bodies(batch.engine, state["out"])
    if kind == "collide":
        w = state["world"]
        w.run_phase(ag2d.PHASE_COLLIDE)
        found = w.read(ag2d.MANIFOLDS, state["out"])
        rows = state["out"].view(np.uint32).reshape(-1, 16)   # views, nothing copied
        return {"count": found.size, "colliders": rows[:, 0:2], "normal_depth": rows[:, 2:5].view(np.float32),
                "count_ids": rows[:, 5:8], "points": rows[:, 8:12].view(np.float32)}
    if kind == "serve":
        server = state["server"]
        ids = [server.submit(w, case["steps"]) for w in state["worlds"]]
        server.wait_all()
        pose = [server.read(r, ag2d.BODY_POSE) for r in ids]
        vy = [server.read(r, ag2d.BODY_VEL_Y) for r in ids]
        for r in ids:
            server.release(r)
        return {"pose": np.concatenate(pose), "vy": np.concatenate(vy)}
    if kind == "query":
        w = state["world"]
        found, touched, dist = [], [], []
        for x, y, h in state["at"]:
            found.append(w.query_aabb((x - h, y - h), (x + h, y + h)))
            i, d = w.query_circle_contacts((x, y), h)
            touched.append(i)
            dist.append(d)
        return {"counts": np.array([a.size for a in found + touched]), "found": _gather(found, state["found"]),
                "touched": _gather(touched, state["touched"]), "distance": _gather(dist, state["distance"])}
    w = state["world"]
    w.step(case["steps"])
    return _read_bodies(w, state["out"])


# ---------------------------------------------------------------------------------------------------------------
# What a pass cannot do without. Per body and step: velocity, position, rotation, timer and state read and written
# (2 x 45 bytes), the collider's shape, offset and material read (about 110 bytes with a polygon's outline), its pose
# and box written (36); about 1.5 contacts a body in a pile, each manifold written with its impulses and last step's
# read (128 bytes). Arithmetic: about 3 candidate pairs a body at 800 operations, 1.5 contacts at 150 operations an
# iteration. A free body: no contacts, 60 operations.
# ---------------------------------------------------------------------------------------------------------------
def _log_uniform_mean(lo, hi):
    return (hi - lo) / math.log(hi / lo) if hi > lo else float(lo)


def work(case):
    kind = case["kind"]
    if kind == "query":
        n = 1.25 * case["bodies"]   # boxes, owners and states of the colliders, read for each of two queries
        return {"bytes": 2.0 * case["queries"] * 21.0 * n, "flops": 2.0 * case["queries"] * 10.0 * n}
    if kind == "collide":
        n = case["bodies"]   # bodies 24, offset 16, shape 50; pose and box written; a pair in four, a manifold in five
        return {"bytes": n * (90.0 + 36.0 + 0.25 * 8.0 + 0.2 * 128.0), "flops": n * (150.0 + 0.25 * 300.0)}
    if kind == "joints":
        n = case["bodies"]
        return {"bytes": case["steps"] * n * (90.0 + 52.0 + 2.0 * 64.0) + 24.0 * n,
                "flops": case["steps"] * n * 2.0 * 8.0 * 120.0}
    if kind == "serve":
        bodies = case["requests"] * _log_uniform_mean(32, case["bodies"])
    elif kind == "flight" or case["worlds"] == 1 or case["scene"] == "capsules":
        bodies = case.get("worlds", 1) * case["bodies"]
    else:
        bodies = case["worlds"] * _log_uniform_mean(16, case["bodies"])
    contacts = 0.0 if kind == "flight" else 1.5
    io = 250.0 + 68.0 * contacts + 28.0   # the saved state in, poses, velocities and states out
    return {"bytes": bodies * (case["steps"] * (90.0 + 110.0 + 36.0 + 128.0 * contacts) + io),
            "flops": bodies * case["steps"] * (60.0 + 1600.0 * contacts + 150.0 * contacts * case.get("iterations", 8))}


def exact(case, seed):
    """Free flight has a closed form; a pile's contacts do not (the order of the impulses decides the result)."""
    if case["kind"] != "flight":
        return None
    s = _flight(case, seed)
    dt = float(np.float32(DT))
    g = np.where(s.mass > 0.0, float(np.float32(GRAVITY)), 0.0)
    t = dt * case["steps"]
    f = lambda a: a.astype(np.float64)
    pose = np.stack([f(s.px) + f(s.vx) * t, f(s.py) + f(s.vy) * t + 0.5 * g * t * t,
                     np.mod(f(s.rot) + f(s.w) * t, 2.0 * math.pi)], axis=1).reshape(-1)
    return {"pose": pose, "vx": f(s.vx), "vy": f(s.vy) + g * t, "spin": f(s.w), "state": None}
