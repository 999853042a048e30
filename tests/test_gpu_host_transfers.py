"""Reads and checkpoints give the same bytes whichever way they travel.

Small packed reads and checkpoints are written by a kernel into page-locked memory, larger ones and other destinations
are copied; alignment and page-locking of the caller's array pick the route. Sizes lie on both sides of the limits
(256 KiB of a packed read: 21,845 poses; 1 MiB of a checkpoint).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ag2d = pytest.importorskip("ag2d")
from ag2d import scenes  # noqa: E402


def _scene(n, k=0):
    side = max(4.0, 3.0 * float(np.sqrt(n)))
    return scenes.make_c1(n, seed=7 + k, width=side, height=side)


@pytest.mark.parametrize("n", [1, 33, 21_844, 21_845, 30_000])
def test_reads_agree_over_destinations(n):
    w = ag2d.World.from_scene(_scene(n))
    w.step(3)
    for field in (ag2d.BODY_POSE, ag2d.BODY_VEL_X, ag2d.BODY_STATE, ag2d.COL_WORLD_X):
        want = w.read(field).view(np.uint8).copy()
        nbytes = want.size
        locked, pageable = ag2d.host_empty(nbytes + 64), np.empty(nbytes + 64, np.uint8)
        for out in (locked[:nbytes], locked[4:4 + nbytes], pageable[:nbytes], pageable[4:4 + nbytes]):
            out[:] = 0xA5
            assert np.array_equal(w.read(field, out).view(np.uint8), want)
        locked[nbytes:] = 0x5A
        w.read(field, locked[:nbytes])
        assert (locked[nbytes:] == 0x5A).all()   # nothing behind the field
    x = w.read(ag2d.BODY_POSE).reshape(-1, 3)
    assert np.array_equal(x[:, 2].view(np.uint32), w.read(ag2d.BODY_ROTATION).view(np.uint32))
    w.close()


@pytest.mark.parametrize("n", [1, 40, 700, 2000, 4000])
def test_checkpoints_agree_over_buffers(n):
    worlds = [ag2d.World.from_scene(_scene(n, k)) for k in range(3)]
    batch = ag2d.Batch(worlds)
    batch.step(20)
    size = batch.save().size
    zeroed = ag2d.host_empty(size)   # the padding between the sections is not written: it keeps what was there
    zeroed[:] = 0
    blob = batch.save(zeroed)
    plain = batch.save(np.zeros(size, np.uint8))
    assert np.array_equal(blob, plain)
    states = []
    for source in (blob, plain):
        batch.load(source)
        assert np.array_equal(batch.save(np.zeros(size, np.uint8)), blob)
        batch.step(5)
        states.append([batch.read(k, f).view(np.uint8).copy() for k in range(3)
                       for f in (ag2d.BODY_COM_X, ag2d.BODY_VEL_Y, ag2d.PREV_MANIFOLDS)])
    assert all(np.array_equal(a, b) for a, b in zip(*states))
