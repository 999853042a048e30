"""A world that the grid solver solves: the steps of a restored engine allocate nothing, the first one included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ag2d = pytest.importorskip("ag2d")
from ag2d import scenes  # noqa: E402


def test_steps_of_a_large_world_allocate_nothing():
    n = 7000
    side = 1.6 * float(np.sqrt(n))
    w = ag2d.World.from_scene(scenes.make_c1(n, seed=3, width=side, height=side), sleep_time=1.0e6)
    batch = ag2d.Batch([w])
    batch.step(24)
    blob = batch.save()
    other = ag2d.Batch.restore(blob)
    allocs = ag2d.device_allocs()
    other.step(3)
    assert ag2d.device_allocs() == allocs
    batch.step(3)
    for f in (ag2d.BODY_POSE, ag2d.BODY_VEL_X, ag2d.BODY_VEL_Y):
        assert np.array_equal(batch.engine.read(f).view(np.uint32), other.engine.read(f).view(np.uint32))
