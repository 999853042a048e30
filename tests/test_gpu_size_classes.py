"""Every size class of the tree builders and solvers gives one world the same bits.

A world's tree is built by one CTA of its size class or by the whole GPU, its contacts are solved by one CTA, by a grid
or by a team of a batch, depending on its size and on the largest world beside it. Worlds at the edges of the classes
(leaves: 256, 1,024, 2,048, 4,096, 5,120, 8,192; solver: 6,912 bodies) are stepped alone, in a batch of their own sizes
(CTA builders) and beside a world too large for those (whole-GPU build with world passes): bodies, manifolds and
impulses are equal bit for bit in all three.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ag2d = pytest.importorskip("ag2d")
from ag2d import scenes  # noqa: E402

SIZES = (1, 2, 31, 256, 257, 1024, 1025, 2048, 2049, 4096, 4097, 5120, 5121, 6911, 6912, 8192, 8193)
STEPS = 24


def _scene(n, k):
    side = max(4.0, 1.6 * float(np.sqrt(n)))   # dense: contacts within a few steps
    return scenes.make_c1(n, seed=100 + k, width=side, height=side)


def _state(engine, k=None):
    read = (lambda f: engine.read(f)) if k is None else (lambda f: engine.read(k, f))
    return [np.ascontiguousarray(read(f)).view(np.uint8) for f in
            (ag2d.BODY_COM_X, ag2d.BODY_COM_Y, ag2d.BODY_VEL_X, ag2d.BODY_VEL_Y, ag2d.BODY_ROTATION,
             ag2d.BODY_ANGULAR_VELOCITY, ag2d.BODY_STATE, ag2d.PREV_MANIFOLDS)]


@pytest.fixture(scope="module")
def alone():
    out = []
    for k, n in enumerate(SIZES):
        w = ag2d.World.from_scene(_scene(n, k))
        w.step(STEPS)
        assert w.counters()["status"] == 0
        out.append(_state(w))
        w.close()
    assert sum(s[-1].size > 0 for s in out) > len(out) // 2   # contacts in most
    return out


@pytest.mark.parametrize("beside", [0, 16_500])
def test_worlds_step_alike_in_every_class(alone, beside):
    worlds = [ag2d.World.from_scene(_scene(n, k)) for k, n in enumerate(SIZES)]
    if beside:
        worlds.append(ag2d.World.from_scene(_scene(beside, 99)))
    batch = ag2d.Batch(worlds)
    batch.step(STEPS)
    assert batch.counters()["status"] == 0
    for k, want in enumerate(alone):
        for i, (a, b) in enumerate(zip(want, _state(batch, k))):
            assert np.array_equal(a, b), (SIZES[k], i)
