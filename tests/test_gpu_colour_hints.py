"""Contacts keep their colours from step to step; a body that gets a mass must not leave two of one colour on it.

Stacks of boxes rest on static platforms. Nothing moves a static body, so its contacts share colours. Some platforms are
then given a mass: in the next step every colour has to be free of contacts that share a movable body, and the solve has
to equal the oracle's FP32 replay of the GPU's own order bit for bit, in the one-CTA solver and in the grid solver (more
than 6,912 bodies). A second world that takes the same commands and one whole step ends at the same bits.
"""
import numpy as np
import pytest

import parity

pytestmark = pytest.mark.gpu

ag2d = pytest.importorskip("ag2d")
from ag2d import scenes  # noqa: E402
from oracle import oraapi  # noqa: E402

COLUMNS = 12   # stacks a platform: fewer contacts than there are first-fit colours
BODY = {"comX": ag2d.BODY_COM_X, "comY": ag2d.BODY_COM_Y, "velocityX": ag2d.BODY_VEL_X, "velocityY": ag2d.BODY_VEL_Y,
        "rotation": ag2d.BODY_ROTATION, "angularVelocity": ag2d.BODY_ANGULAR_VELOCITY, "invMass": ag2d.BODY_INV_MASS,
        "invInertia": ag2d.BODY_INV_INERTIA}
MOVED = (ag2d.BODY_VEL_X, ag2d.BODY_VEL_Y, ag2d.BODY_ANGULAR_VELOCITY, ag2d.BODY_COM_X, ag2d.BODY_COM_Y)


def _stacks(platforms, high):
    """Platforms first (bodies 0 .. platforms - 1), then their boxes, resting from the start."""
    b = scenes._Builder([scenes.FRICTION_MATERIAL])
    x = [20.0 * (p % 40) for p in range(platforms)]
    y = [20.0 * (p // 40) for p in range(platforms)]
    for p in range(platforms):
        b.add(scenes.BOX, x[p], y[p] - 0.5, width=1.2 * COLUMNS, height=1.0, mass=0.0)
    for p in range(platforms):
        for c in range(COLUMNS):
            for k in range(high):
                b.add(scenes.BOX, x[p] + 1.1 * (c - 0.5 * (COLUMNS - 1)), y[p] + 0.5 + k, width=1.0, height=1.0, mass=1.0)
    w = ag2d.World(dt=1.0 / 60.0, sleep_time=1.0e6)
    return w, w.add_scene(b.build("stacks"))


def _command(w, handles, platforms, kind):
    for p in range(0, platforms, 2):
        if kind == "mass":
            w.set_body_mass(int(handles[p]), 30.0)
        elif kind == "density":
            w.set_body_mass_from_density(int(handles[p]), 2.0)
        else:   # a mass, none and another before one step
            for m in (30.0, 0.0, 12.0):
                w.set_body_mass(int(handles[p]), m)


def _oracle(w):
    """The oracle's world with the state the solver reads; what it does not read is left at zero."""
    nb, nc = w.counts()
    d = {"body." + k: w.read(f) for k, f in BODY.items()}
    for k in set(oraapi.OraWorld.BODY_F.values()) - set(BODY):
        d["body." + k] = np.zeros(nb, np.float32)
    d["body.islandId"] = np.zeros(nb, np.uint32)
    for k in oraapi.OraWorld.COL_F.values():
        d["col." + k] = np.zeros(nc, np.float32)
    for k in oraapi.OraWorld.COL_U.values():
        d["col." + k] = np.zeros(nc, np.uint32)
    d["col.bodyIndex"] = w.read(ag2d.COL_BODY)
    d["col.materialIndex"] = np.ones(nc, np.uint32)
    for k in ("circle.radius", "box.halfWidth", "box.halfHeight", "poly.vertices", "poly.normals"):
        d[k] = np.zeros(0, np.float32)
    d["poly.counts"] = np.zeros(0, np.uint32)
    d["body.groupStarts"], d["col.groupStarts"] = np.array([0, 0, 0, nb]), np.array([0, 0, 0, nc])
    return oraapi.OraWorld(d, "", list(oraapi.DEFAULT_MATERIALS)[:1] + [scenes.FRICTION_MATERIAL]), d


def _to_oracle(m):
    out = np.zeros(m.shape[0], oraapi.MANIFOLD_DTYPE)
    for f in ("a", "b", "nx", "ny", "depth", "count"):
        out[f] = m[f]
    for f in ("px", "py", "id", "jn", "jt"):
        out[f] = np.stack([m[f + "0"], m[f + "1"]], 1)
    return out


@pytest.mark.parametrize("kind", ["mass", "density", "twice"])
@pytest.mark.parametrize("platforms,high", [(24, 2), (300, 2)])
def test_a_body_that_gets_a_mass_is_solved_in_order(platforms, high, kind):
    worlds = [_stacks(platforms, high) for _ in range(2)]
    for w, handles in worlds:
        w.step(8)   # every contact is there and keeps its colour
        assert w.read(ag2d.PREV_MANIFOLDS).size >= platforms * COLUMNS * high
        _command(w, handles, platforms, kind)
    w, handles = worlds[0]
    w.flush_commands()
    for phase in (ag2d.PHASE_INTEGRATE, ag2d.PHASE_SPATIAL_FULL, ag2d.PHASE_BROAD, ag2d.PHASE_NARROW):
        w.run_phase(phase)
    m_in = _to_oracle(w.read(ag2d.MANIFOLDS))
    ora, d = _oracle(w)
    assert np.count_nonzero(d["body.invMass"][:platforms]) == (platforms + 1) // 2
    w.run_phase(ag2d.PHASE_SOLVE)
    order, starts = w.read(ag2d.SOLVE_ORDER).astype(np.int64), w.read(ag2d.COLOR_STARTS)
    assert np.array_equal(np.sort(order), np.arange(m_in.size))
    body, inv_mass = d["col.bodyIndex"], d["body.invMass"]
    for c in range(starts.size - 1):
        ms = order[starts[c]:starts[c + 1]]
        bodies = np.concatenate([body[m_in["a"][ms]], body[m_in["b"][ms]]])
        dyn = bodies[inv_mass[bodies] > 0]
        assert np.unique(dyn).size == dyn.size, f"colour {c} shares a movable body"
    rep = ora.solve(m_in, order)
    ours = _to_oracle(w.read(ag2d.MANIFOLDS))
    assert parity.mismatches(ours["jn"], rep["jn"]) == 0
    assert parity.mismatches(ours["jt"], rep["jt"]) == 0
    for field, ref in zip(MOVED, ("velX", "velY", "angVel", "comX", "comY")):
        assert parity.mismatches(w.read(field), ora.a[ref]) == 0, ref
    other, _ = worlds[1]
    other.step(1)
    assert other.counters()["status"] == 0
    for field in MOVED:
        assert parity.mismatches(w.read(field), other.read(field)) == 0
