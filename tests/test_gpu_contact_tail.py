"""A movable body with more contacts than there are colours: the rest are solved one after the other, in every solver.

A beam under hundreds of boxes, and a static ground that is given a mass under its boxes, exhaust the colours. Each solve
equals the oracle's FP32 replay of its own order bit for bit (one CTA; the grid, with more than 6,912 bodies), and a batch
of such worlds (team solver, plain and pipelined, records in global and in shared memory) ends at the bits of each alone.
"""
import numpy as np
import pytest

import parity
from test_gpu_colour_hints import MOVED, _oracle, _to_oracle

pytestmark = pytest.mark.gpu

ag2d = pytest.importorskip("ag2d")
from ag2d import scenes  # noqa: E402

LAST_COLOR = 255


def _beam(boxes, others=0, mass=50.0):
    b = scenes._Builder([scenes.FRICTION_MATERIAL])
    length = 0.55 * boxes
    for k in range(5):
        b.add(scenes.BOX, -0.5 * length + 0.25 * k * length, -1.0, width=1.0, height=1.0, mass=0.0)
    b.add(scenes.BOX, 0.0, 0.0, width=length + 2.0, height=1.0, mass=mass)
    for k in range(boxes):
        b.add(scenes.BOX, 0.55 * (k - 0.5 * (boxes - 1)), 0.749, width=0.5, height=0.5, mass=0.2)
    for k in range(others):
        b.add(scenes.CIRCLE, 500.0 + 3.0 * (k % 100), 500.0 + 3.0 * (k // 100), radius=0.5, mass=1.0)
    w = ag2d.World(dt=1.0 / 60.0, sleep_time=1.0e6)
    return w, w.add_scene(b.build("beam"))


def _solve_against_the_replay(w):
    for phase in (ag2d.PHASE_INTEGRATE, ag2d.PHASE_SPATIAL_FULL, ag2d.PHASE_BROAD, ag2d.PHASE_NARROW):
        w.run_phase(phase)
    m_in = _to_oracle(w.read(ag2d.MANIFOLDS))
    ora, d = _oracle(w)
    w.run_phase(ag2d.PHASE_SOLVE)
    order, starts = w.read(ag2d.SOLVE_ORDER).astype(np.int64), w.read(ag2d.COLOR_STARTS)
    assert np.array_equal(np.sort(order), np.arange(m_in.size)) and starts[-1] == m_in.size
    body, inv_mass = d["col.bodyIndex"], d["body.invMass"]
    for c in range(min(starts.size - 1, LAST_COLOR)):
        ms = order[starts[c]:starts[c + 1]]
        bodies = np.concatenate([body[m_in["a"][ms]], body[m_in["b"][ms]]])
        dyn = bodies[inv_mass[bodies] > 0]
        assert np.unique(dyn).size == dyn.size, f"colour {c} shares a movable body"
    tail = order[starts[LAST_COLOR]:] if starts.size > LAST_COLOR + 1 else order[:0]
    assert np.all(np.diff(tail) > 0)
    rep = ora.solve(m_in, order)
    ours = _to_oracle(w.read(ag2d.MANIFOLDS))
    assert parity.mismatches(ours["jn"], rep["jn"]) == 0
    assert parity.mismatches(ours["jt"], rep["jt"]) == 0
    for field, ref in zip(MOVED, ("velX", "velY", "angVel", "comX", "comY")):
        assert parity.mismatches(w.read(field), ora.a[ref]) == 0, ref
    return tail.size


# 191 contacts of one body take a colour in the rounds; after some steps up to 64 more have kept theirs.
@pytest.mark.parametrize("steps,boxes,others", [(2, 190, 0), (2, 200, 0), (2, 600, 0), (2, 200, 7000), (2, 600, 7000),
                                                (0, 180, 0), (0, 200, 0), (0, 200, 7000)])
def test_a_beam_with_more_contacts_than_colours(steps, boxes, others):
    w, _ = _beam(boxes, others)
    w.step(steps)
    assert (_solve_against_the_replay(w) > 0) == (boxes > (255 if steps else 191))
    w.step(2)
    assert w.counters()["status"] == 0


@pytest.mark.parametrize("boxes,others", [(700, 0), (700, 7000)])
def test_a_ground_that_gets_a_mass_under_its_boxes(boxes, others):
    w, handles = _beam(boxes, others, mass=0.0)
    other, other_handles = _beam(boxes, others, mass=0.0)
    for world, hs in ((w, handles), (other, other_handles)):
        world.step(8)
        world.set_body_mass(int(hs[5]), 400.0)
    w.flush_commands()
    assert _solve_against_the_replay(w) > 0
    other.step(1)
    for f in MOVED:
        assert parity.mismatches(w.read(f), other.read(f)) == 0
    other.step(20)
    assert other.counters()["status"] == 0


@pytest.mark.parametrize("on_chip", [0, 1])
@pytest.mark.parametrize("big_mode", [0, 2])
def test_batches_of_such_worlds(big_mode, on_chip):
    sizes = (210, 3, 450, 1500)   # two within a team of 512 colliders, one larger, one between them
    alone = []
    for n in sizes:
        w, _ = _beam(n)
        w.step(3)
        alone.append([w.read(f).view(np.uint32) for f in MOVED])
    batch = ag2d.Batch([_beam(n)[0] for n in sizes])
    batch.engine.set_tuning({"team_colliders": 512, "team_threads": 128, "big_team_mode": big_mode,
                             "team_cons_on_chip": on_chip, "query_threads": 256, "narrow_threads": 256})
    batch.step(3)
    assert batch.counters()["status"] == 0
    for k, want in enumerate(alone):
        for f, a in zip(MOVED, want):
            assert np.array_equal(batch.read(k, f).view(np.uint32), a), (sizes[k], f)


@pytest.mark.parametrize("n,steps", [(800, 260), (7200, 120)])
def test_a_settled_pile_whose_ground_gets_a_mass(n, steps):
    """With sleepers on the ground in the smaller pile: they wake and bring their stored contacts."""
    worlds = []
    for _ in range(2):
        w = ag2d.World()
        side = 1.6 * float(np.sqrt(n))
        handles = w.add_scene(scenes.make_c1(n, seed=n, width=side, height=side))
        w.step(steps)
        w.set_body_mass(int(handles[0]), 5000.0)
        worlds.append(w)
    w, other = worlds
    ground = int(np.argmin(w.read(ag2d.BODY_INV_MASS)))
    w.flush_commands()
    w.run_phase(ag2d.PHASE_INTEGRATE)
    for phase in (ag2d.PHASE_SPATIAL_FULL, ag2d.PHASE_BROAD, ag2d.PHASE_NARROW, ag2d.PHASE_WAKE):
        w.run_phase(phase)
    m_in = _to_oracle(w.read(ag2d.MANIFOLDS))
    ora, d = _oracle(w)
    body = d["col.bodyIndex"]
    assert d["body.invMass"][ground] > 0
    assert np.count_nonzero((body[m_in["a"]] == ground) | (body[m_in["b"]] == ground)) > 20
    w.run_phase(ag2d.PHASE_SOLVE)
    order = w.read(ag2d.SOLVE_ORDER).astype(np.int64)
    assert np.array_equal(np.sort(order), np.arange(m_in.size))
    rep = ora.solve(m_in, order)
    ours = _to_oracle(w.read(ag2d.MANIFOLDS))
    assert parity.mismatches(ours["jn"], rep["jn"]) == 0
    for field, ref in zip(MOVED, ("velX", "velY", "angVel", "comX", "comY")):
        assert parity.mismatches(w.read(field), ora.a[ref]) == 0, ref
    other.step(1)
    assert other.counters()["status"] == 0
    for f in MOVED:
        assert parity.mismatches(w.read(f), other.read(f)) == 0
    other.step(10)
    assert other.counters()["status"] == 0
