"""Contacts that need more colours than the 64 first-fit ones, and the two single-world solvers against each other.

A beam with many small boxes on it needs a colour for each of them. With few bodies one CTA solves the world, with more
than 6,912 the grid does; either solve equals the oracle's FP32 replay of its own order bit for bit. In a process where
the grid solves every single world (AG2D_SOLVER=grid), worlds of any size end at the bits that the one-CTA solver gives.
"""
import hashlib
import os
import subprocess
import sys

import numpy as np
import pytest

import parity
from test_gpu_colour_hints import MOVED, _oracle, _to_oracle

pytestmark = pytest.mark.gpu

ag2d = pytest.importorskip("ag2d")
from ag2d import scenes  # noqa: E402

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _beam(boxes, others):
    """A beam lying on static supports, the boxes on it, and bodies that touch nothing."""
    b = scenes._Builder([scenes.FRICTION_MATERIAL])
    length = 0.55 * boxes
    for k in range(5):
        b.add(scenes.BOX, -0.5 * length + 0.25 * k * length, -1.0, width=1.0, height=1.0, mass=0.0)
    b.add(scenes.BOX, 0.0, 0.0, width=length + 2.0, height=1.0, mass=50.0)
    for k in range(boxes):
        b.add(scenes.BOX, 0.55 * (k - 0.5 * (boxes - 1)), 0.75, width=0.5, height=0.5, mass=0.2)
    for k in range(others):
        b.add(scenes.CIRCLE, 500.0 + 3.0 * (k % 100), 500.0 + 3.0 * (k // 100), radius=0.5, mass=1.0)
    w = ag2d.World(dt=1.0 / 60.0, sleep_time=1.0e6)
    w.add_scene(b.build("beam"))
    return w


# Up to one, two and three words of colours above the first 64; 70 with kept colours from several steps.
@pytest.mark.parametrize("boxes,others,steps", [(70, 0, 6), (70, 7000, 6), (120, 7000, 2), (150, 7000, 2),
                                                (180, 0, 2), (180, 7000, 2)])
def test_many_colours_are_solved_in_order(boxes, others, steps):
    w = _beam(boxes, others)
    w.step(steps)
    for phase in (ag2d.PHASE_INTEGRATE, ag2d.PHASE_SPATIAL_DYNAMIC, ag2d.PHASE_BROAD, ag2d.PHASE_NARROW):
        w.run_phase(phase)
    m_in = _to_oracle(w.read(ag2d.MANIFOLDS))
    assert m_in.size >= boxes
    ora, _ = _oracle(w)
    w.run_phase(ag2d.PHASE_SOLVE)
    order, starts = w.read(ag2d.SOLVE_ORDER).astype(np.int64), w.read(ag2d.COLOR_STARTS)
    assert starts.size - 1 >= boxes and starts[-1] == m_in.size
    assert np.array_equal(np.sort(order), np.arange(m_in.size))
    rep = ora.solve(m_in, order)
    ours = _to_oracle(w.read(ag2d.MANIFOLDS))
    assert parity.mismatches(ours["jn"], rep["jn"]) == 0
    assert parity.mismatches(ours["jt"], rep["jt"]) == 0
    for field, ref in zip(MOVED, ("velX", "velY", "angVel", "comX", "comY")):
        assert parity.mismatches(w.read(field), ora.a[ref]) == 0, ref


def _digests():
    """Name and digest of the state after some steps, for worlds that one CTA solves unless told otherwise."""
    out = []
    for n in (1, 31, 257, 2048, 6912):
        side = max(4.0, 1.6 * float(np.sqrt(n)))
        out.append((f"dense {n}", ag2d.World.from_scene(scenes.make_c1(n, seed=n, width=side, height=side)), 24))
    out.append(("beam", _beam(150, 0), 8))
    # From the one CTA's share of contacts (4,096) to more and back, as the bodies land and spread.
    out.append(("landing", ag2d.World.from_scene(scenes.make_c1(5000, seed=9, width=160.0, height=80.0)), 150))
    for name, w, steps in out:
        w.step(steps)
        assert w.counters()["status"] == 0
        h = hashlib.sha256()
        for f in MOVED + (ag2d.BODY_STATE, ag2d.BODY_SLEEP_ISLAND, ag2d.PREV_MANIFOLDS):
            h.update(np.ascontiguousarray(w.read(f)).tobytes())
        yield f"{name} {h.hexdigest()}"


def test_grid_and_one_cta_agree():
    code = "import sys; sys.path[:0] = %r\nimport test_gpu_many_colours as t\nprint('\\n'.join(t._digests()))" % (
        [os.path.join(ROOT, "tests"), os.path.join(ROOT, "physicssimulation-agony_b200"), ROOT],)
    r = subprocess.run([sys.executable, "-c", code], env={**os.environ, "AG2D_SOLVER": "grid"}, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.strip().split("\n") == list(_digests())
