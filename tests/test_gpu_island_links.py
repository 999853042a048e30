"""The islands phase after a wake that came after the solve: bodies that the wake brought in are linked.

Two boxes sleep on the ground, one on the other, and a third falls on them. The phases run one by one, the wake after the
solve: the sleeping pair and its stored contacts join the falling body's island, which moves, so none of them may fall
asleep again. (The one-CTA solver links the islands of what it solved, where the pair was not awake yet.)
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ag2d = pytest.importorskip("ag2d")
from ag2d import scenes  # noqa: E402


def test_a_wake_after_the_solve_links_what_it_woke():
    b = scenes._Builder([scenes.FRICTION_MATERIAL])
    b.add(scenes.BOX, 0.0, -0.5, width=20.0, height=1.0, mass=0.0)
    b.add(scenes.BOX, 0.0, 0.49, width=1.0, height=1.0, mass=1.0)
    b.add(scenes.BOX, 0.0, 1.47, width=1.0, height=1.0, mass=1.0)
    b.add(scenes.BOX, 0.0, 12.0, vy=-3.0, width=1.0, height=1.0, mass=1.0)
    w = ag2d.World(dt=1.0 / 60.0, sleep_speed=0.5, sleep_time=0.01)
    w.add_scene(b.build("drop on sleepers"))
    w.step(10)
    assert w.read(ag2d.BODY_STATE).tolist() == [0, 1, 1, 2]
    for _ in range(200):
        for phase in (ag2d.PHASE_INTEGRATE, ag2d.PHASE_SPATIAL_DYNAMIC, ag2d.PHASE_BROAD, ag2d.PHASE_NARROW,
                      ag2d.PHASE_SOLVE, ag2d.PHASE_WAKE):
            w.run_phase(phase)
        woke = w.counters()["woke"]
        if woke:
            break
    assert woke == 2 and abs(float(w.read(ag2d.BODY_VEL_Y)[3])) > 0.5
    w.run_phase(ag2d.PHASE_ISLANDS)
    assert w.read(ag2d.BODY_STATE).tolist() == [0, 2, 2, 2]
