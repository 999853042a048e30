"""Jointed worlds of a batch whose bodies fall asleep and wake: every world's constraints keep the order they have alone.

The active constraints are solved in an order that the swaps between the groups (inactive, sleeping, active) decide. Worlds
with chains that settle at different times and are woken by falling balls, each bit for bit as alone at every look.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ag2d = pytest.importorskip("ag2d")
from ag2d import scenes  # noqa: E402

FIELDS = (ag2d.BODY_POSE, ag2d.BODY_VEL_X, ag2d.BODY_VEL_Y, ag2d.BODY_ANGULAR_VELOCITY, ag2d.BODY_STATE)


def _world(k):
    rng = np.random.default_rng(50 + k)
    w = ag2d.World(sleep_speed=0.4, sleep_time=0.2)
    mat = w.add_material(*scenes.FRICTION_MATERIAL)
    w.add_collider(w.create_body(0.0, -1.0, mass=0.0, inertia=0.0), scenes.BOX, width=80.0, height=2.0, material=mat)
    for c in range(3 + k):
        links = []
        for i in range(4 + c):
            b = w.create_body(-30.0 + 9.0 * c + 0.7 * i, 0.31 + 0.15 * c, mass=1.0, inertia=0.2)
            w.add_collider(b, scenes.CIRCLE, radius=0.3, material=mat)
            if links and i % 3 == 2:
                w.create_spring(links[-1], b, (0.0, 0.0), (0.0, 0.0), 0.7, 60.0, 6.0)
            elif links:
                w.create_revolute_joint(links[-1], b, (0.35, 0.0), (-0.35, 0.0), 4.0e3, 40.0)
            links.append(b)
        if c % 2:
            w.create_motor(links[0], 0.0, 3.0)
    for _ in range(3):   # balls that come down on sleeping chains later
        ball = w.create_body(float(rng.uniform(-28, 10)), float(rng.uniform(10, 40)), mass=2.0, inertia=0.4)
        w.add_collider(ball, scenes.CIRCLE, radius=0.5, material=mat)
    return w


def test_each_world_steps_as_alone_through_sleep_and_wake():
    worlds = 4
    alone = [_world(k) for k in range(worlds)]
    batch = ag2d.Batch([_world(k) for k in range(worlds)])
    slept = woke = 0
    for _ in range(60):
        batch.step(5)
        for k, w in enumerate(alone):
            w.step(5)
            slept += w.counters()["slept"]
            woke += w.counters()["woke"]
            for f in FIELDS:
                assert np.array_equal(batch.read(k, f).view(np.uint32), w.read(f).view(np.uint32)), (k, f)
    assert slept > 0 and woke > 0
