"""Requests that join the server together with one for no steps: the round makes no step, and what the others need in their
first step (every collider posed, the static ones among them) is still owed to them in the next round.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ag2d = pytest.importorskip("ag2d")
from ag2d import scenes  # noqa: E402


def _world(n, ccd):
    side = 1.6 * max(4.0, float(np.sqrt(n)))
    return ag2d.World.from_scene(scenes.make_c1(n, seed=n, width=side, height=side), ccd=ccd)


@pytest.mark.parametrize("ccd", [False, True])
@pytest.mark.parametrize("sizes", [(60, 3), (60, 3, 200, 9), (3, 60)])
def test_requests_beside_one_for_no_steps(sizes, ccd):
    steps = 30
    # The first request is larger than the budget and runs alone; the others wait and join in one round.
    server = ag2d.Server(memory_budget_bytes=6 << 20, steps_per_round=4, ccd=ccd)
    first = server.submit(_world(6000, ccd), 60)
    ids = [(n, 0 if n == 3 else steps, server.submit(_world(n, ccd), 0 if n == 3 else steps)) for n in sizes]
    server.wait_all()
    for n, k, r in ids:
        alone = _world(n, ccd)
        alone.step(k)
        for f in (ag2d.BODY_POSE, ag2d.BODY_VEL_Y, ag2d.BODY_STATE):
            assert np.array_equal(server.read(r, f).view(np.uint32), alone.read(f).view(np.uint32)), (n, f)
    server.release(first)
