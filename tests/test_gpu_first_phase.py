"""A phase as the first thing a world does: its counters start at zero, whatever the memory held before."""
import pytest

pytestmark = pytest.mark.gpu

ag2d = pytest.importorskip("ag2d")
from ag2d import scenes  # noqa: E402


@pytest.mark.parametrize("phase", [ag2d.PHASE_SPATIAL_FULL, ag2d.PHASE_SPATIAL_DYNAMIC, ag2d.PHASE_INTEGRATE])
def test_a_phase_run_first(phase):
    for k in range(40):
        used = ag2d.World.from_scene(scenes.make_c1(30 + 7 * k, seed=k, width=8.0, height=8.0))
        used.step(3)
        used.close()   # leaves its small buffers' contents to the next engine
        w = ag2d.World.from_scene(scenes.make_c1(20, seed=k, width=8.0, height=8.0))
        w.run_phase(phase)
        c = w.counters()
        assert all(c[n] == 0 for n in ("status", "pairs", "manifolds", "colors", "woke", "slept", "events", "stored"))
        w.close()
