"""The two schedules of the constraint solver give the same bits.

Sets whose bodies fit shared memory are solved as a dataflow over per-body versions; larger ones with a block barrier
after every level. Bodies bound by no common constraint do not act on one another, so a graph of constraints solved by
itself (dataflow) and beside 6,000 motors on bodies of their own (too many bodies: barriers) must move its bodies
alike, bit for bit: both schedules apply each body's updates in dense order.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ag2d = pytest.importorskip("ag2d")

FIELDS = (ag2d.BODY_COM_X, ag2d.BODY_COM_Y, ag2d.BODY_VEL_X, ag2d.BODY_VEL_Y, ag2d.BODY_ROTATION,
          ag2d.BODY_ANGULAR_VELOCITY)


def _run(n, joints, filler, iterations):
    rng = np.random.default_rng(n)
    w = ag2d.World(dt=1.0 / 60.0, sleep_time=1.0e6)
    w.add_collider(w.create_body(0.0, -1000.0, mass=0.0, inertia=0.0), 1, width=10.0, height=1.0)
    bodies = [w.create_body(float(rng.uniform(-50, 50)), float(rng.uniform(0, 100)), vx=float(rng.normal()),
                            vy=float(rng.normal()), w=float(rng.normal(0, 0.5)),
                            mass=0.0 if i % 7 == 3 else float(rng.uniform(0.5, 3.0)),
                            inertia=0.0 if i % 7 == 3 else float(rng.uniform(0.05, 1.0))) for i in range(n)]
    for j in range(joints):
        kind = (ag2d.JOINT_SPRING, ag2d.JOINT_REVOLUTE, ag2d.JOINT_PRISMATIC, ag2d.JOINT_SLIDER,
                ag2d.JOINT_MOTOR)[j % 5]
        a, b = (rng.integers(n), rng.integers(n))
        lo = float(rng.uniform(-3, 0))
        if kind == ag2d.JOINT_MOTOR or a == b:
            w.create_joint(ag2d.JOINT_MOTOR, bodies[a], 0, target_speed=float(rng.uniform(-3, 3)),
                           max_torque=float(rng.uniform(0.5, 20)))
        else:
            w.create_joint(kind, bodies[a], bodies[b], tuple(rng.uniform(-0.5, 0.5, 2).tolist()),
                           tuple(rng.uniform(-0.5, 0.5, 2).tolist()), rest_length=float(rng.uniform(0.5, 5.0)),
                           stiffness=float(rng.uniform(20, 300)), damping=float(rng.uniform(0.5, 8.0)),
                           axis=tuple(rng.normal(0, 1, 2).tolist()), limits=(lo, lo + 2.0), enable_limit=bool(j % 3))
    for i in range(filler):
        b = w.create_body(500.0 + i, 0.0, mass=1.0, inertia=0.5)
        w.create_joint(ag2d.JOINT_MOTOR, b, 0, target_speed=1.0, max_torque=1.0)
    for kind, it in zip((ag2d.JOINT_SPRING, ag2d.JOINT_REVOLUTE, ag2d.JOINT_PRISMATIC), iterations):
        w.set_joint_iterations(kind, it)
    w.step(8)
    assert w.counters()["status"] == 0
    rows = [w.body_index(h) for h in bodies]
    out = np.stack([w.read(f)[rows] for f in FIELDS]).astype(np.float32)
    w.close()
    return out.view(np.uint32)


# One body; a warp and one; more constraints of a type than the block has threads; long chains on few bodies; types
# with iterations of their own.
@pytest.mark.parametrize("n,joints,iterations", [(1, 1, (8, 8, 8)), (33, 40, (8, 8, 8)), (1500, 6000, (8, 8, 8)),
                                                 (3, 200, (8, 8, 8)), (300, 900, (3, 7, 1))])
def test_dataflow_and_barriers_agree(n, joints, iterations):
    alone, beside = _run(n, joints, 0, iterations), _run(n, joints, 6000, iterations)
    assert np.array_equal(alone, beside)
