"""The narrow phase's two polygon searches give the same manifolds.

Large sets of mostly polygons search their polygon pairs one a lane (up to eight vertices) where a warp has enough of
them and in groups of lanes otherwise; blocks of 512 threads always search in groups. Both evaluate the same expressions
and keep the same axis on ties, so the manifolds must be equal bit for bit: over triangles to 16-gons, exact duplicates
in position and rotation, identical shapes (ties everywhere), and other shapes between them.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ag2d = pytest.importorskip("ag2d")
from ag2d import scenes  # noqa: E402


def _scene(n, most, polygons):
    rng = np.random.default_rng(n + most)
    b = scenes._Builder([scenes.FRICTION_MATERIAL])
    side = 0.9 * math.sqrt(n)
    square = np.array([[-0.5, -0.5], [0.5, -0.5], [0.5, 0.5], [-0.5, 0.5]], np.float32)
    for i in range(n):
        x, y = float(rng.uniform(0, side)), float(rng.uniform(0, side))
        if i % 5 == 4:   # a lattice of equal squares, axis-aligned: equal overlaps on several axes
            b.add(scenes.POLYGON, round(x * 2) / 2, round(y * 2) / 2, mass=1.0, verts=square)
        elif rng.random() < polygons:
            verts = scenes.polygon_on_circle(rng, float(rng.uniform(0.4, 0.9)), 3, most)
            b.add(scenes.POLYGON, x, y, rot=float(rng.uniform(0, 6)), mass=1.0, verts=verts)
        elif i % 2:
            b.add(scenes.BOX, x, y, rot=float(rng.uniform(0, 6)), mass=1.0, width=0.8, height=0.5)
        else:
            b.add(scenes.CIRCLE, x, y, mass=1.0, radius=0.4)
    return b.build("narrow_forms")


@pytest.mark.parametrize("n,most,polygons", [(20_000, 8, 1.0), (20_000, 16, 1.0), (24_000, 9, 0.6)])
def test_lanes_and_groups_agree(n, most, polygons):
    out = []
    for threads in (256, 128, 512):
        w = ag2d.World.from_scene(_scene(n, most, polygons))
        tuning = {name: 0 for name, _ in ag2d.Tuning._fields_}
        w.set_tuning({**tuning, "query_threads": 128, "narrow_threads": threads})
        for _ in range(2):   # the second pass sizes its launch by the first one's pairs
            w.run_phase(ag2d.PHASE_COLLIDE)
        c = w.counters()
        assert c["status"] == 0 and c["pairs"] > 40_000
        out.append(np.ascontiguousarray(w.read(ag2d.MANIFOLDS)).view(np.uint8))
        w.close()
    assert out[0].size > 0
    assert np.array_equal(out[0], out[2]) and np.array_equal(out[1], out[2])
