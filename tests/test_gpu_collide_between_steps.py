"""Collision passes (AG2D_PHASE_COLLIDE) between steps, replayed from a graph or not: the pass finds what the phases one by
one find, and the steps go on as without it. A step trades the buffer that a captured pass writes its manifolds into.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ag2d = pytest.importorskip("ag2d")
from ag2d import scenes  # noqa: E402

STATE = (ag2d.BODY_POSE, ag2d.BODY_VEL_X, ag2d.BODY_VEL_Y, ag2d.BODY_ANGULAR_VELOCITY, ag2d.BODY_STATE,
         ag2d.PREV_MANIFOLDS)


def _world(n):
    side = 1.6 * float(np.sqrt(n))
    return ag2d.World.from_scene(scenes.make_c1(n, seed=n, width=side, height=side), sleep_time=1.0e6)


@pytest.mark.parametrize("n", [300, 6000, 20000])   # trees by one CTA and by the whole GPU
@pytest.mark.parametrize("passes", [1, 3])
def test_collision_passes_between_steps(n, passes):
    plain, phases, w = _world(n), _world(n), _world(n)
    for x in (plain, phases, w):
        x.step(6)
    for steps in (0, 1, 1, 2, 1):
        for x in (plain, phases, w):
            x.step(steps)
        for phase in (ag2d.PHASE_SPATIAL_DYNAMIC, ag2d.PHASE_BROAD):
            phases.run_phase(phase)
        want = phases.read(ag2d.PAIRS)
        for _ in range(passes):
            w.run_phase(ag2d.PHASE_COLLIDE)
            assert np.array_equal(w.read(ag2d.PAIRS), want)
        found = w.read(ag2d.MANIFOLDS)
        phases.run_phase(ag2d.PHASE_NARROW)
        expect = phases.read(ag2d.MANIFOLDS).copy()
        for f in ("jn0", "jt0", "jn1", "jt1"):   # a collision pass does not warm-start
            expect[f] = 0.0
        assert found.tobytes() == expect.tobytes()
    for x in (plain, w):
        x.step(3)
    for f in STATE:
        a, b = plain.read(f), w.read(f)
        assert a.tobytes() == b.tobytes()
    assert w.counters()["retries"] == 0


def test_passes_of_a_batch_between_steps():
    """Three hundred worlds, one of them too large for the tree builders of one CTA: two sort passes on the world ids."""
    def batch():
        rng = np.random.default_rng(7)
        return ag2d.Batch([_world(int(k)) for k in np.append(rng.integers(1, 40, 299), 16_500)])
    plain, b = batch(), batch()
    for x in (plain, b):
        x.step(4)
    for _ in range(3):
        for _ in range(4):
            b.engine.run_phase(ag2d.PHASE_COLLIDE)
        for x in (plain, b):
            x.step(1)
    for f in STATE:
        assert plain.engine.read(f).tobytes() == b.engine.read(f).tobytes()
    first = None
    for _ in range(4):
        b.engine.run_phase(ag2d.PHASE_COLLIDE)
        got = (b.engine.read(ag2d.DYN_SORTED).tobytes(), b.engine.read(ag2d.MANIFOLDS).tobytes())
        first = first or got
        assert got == first


def test_passes_of_a_batch_with_one_world_pass():
    """As above with few worlds: one sort pass on the world ids, an odd number in all."""
    def batch():
        return ag2d.Batch([_world(n) for n in (40, 16_500, 300)])
    plain, b = batch(), batch()
    for x in (plain, b):
        x.step(4)
    first = None
    for _ in range(4):
        b.engine.run_phase(ag2d.PHASE_COLLIDE)
        got = (b.engine.read(ag2d.DYN_SORTED).tobytes(), b.engine.read(ag2d.MANIFOLDS).tobytes())
        first = first or got
        assert got == first
    for x in (plain, b):
        x.step(2)
    for f in STATE:
        assert plain.engine.read(f).tobytes() == b.engine.read(f).tobytes()


@pytest.mark.parametrize("n", [40, 3000])
@pytest.mark.parametrize("edit", [False, True])
def test_a_pass_before_the_first_step(n, edit):
    """The static colliders have no poses yet (or a static body was moved since): the pass poses them, and the step after it
    does not take over a tree from before. 'edit': the pass follows a command on the ground instead of the creation."""
    def world():
        b = scenes._Builder([scenes.FRICTION_MATERIAL])
        b.add(scenes.BOX, 0.0, -0.5, width=3.0 * n, height=1.0, mass=0.0)
        for k in range(n):
            b.add(scenes.BOX, 1.1 * (k - 0.5 * n), 0.499, width=1.0, height=1.0, mass=1.0)
        w = ag2d.World(sleep_time=1.0e6)
        ground = int(w.add_scene(b.build("row"))[0])
        if edit:
            w.step(2)
            w.set_body_position(ground, 0.0, -0.45)
            w.flush_commands()
        return w
    plain, phases, w = world(), world(), world()
    for phase in (ag2d.PHASE_SPATIAL_FULL, ag2d.PHASE_SPATIAL_DYNAMIC, ag2d.PHASE_BROAD):
        phases.run_phase(phase)
    for _ in range(3):
        w.run_phase(ag2d.PHASE_COLLIDE)
        assert np.array_equal(w.read(ag2d.PAIRS), phases.read(ag2d.PAIRS))
    assert w.read(ag2d.MANIFOLDS).size >= n   # every box on the ground
    for x in (plain, w):
        x.step(6)
    for f in STATE:
        assert plain.read(f).tobytes() == w.read(f).tobytes()
