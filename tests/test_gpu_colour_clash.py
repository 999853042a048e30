"""Colours to keep that two contacts on one movable body share: the step is made as if no colour were kept.

A checkpoint carries the colours of the last step's contacts. One whose colours were all set alike is loaded, and steps
as the same checkpoint without colours does, bit for bit: in the one-CTA solver, the grid solver (more than 6,912
bodies) and the team solver of a batch.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ag2d = pytest.importorskip("ag2d")
from ag2d import scenes  # noqa: E402

SECTIONS, PREVCOLOR = 29, 24
FIELDS = (ag2d.BODY_POSE, ag2d.BODY_VEL_X, ag2d.BODY_VEL_Y, ag2d.BODY_ANGULAR_VELOCITY, ag2d.BODY_STATE)


class _Header(ctypes.Structure):
    _fields_ = [("magic", ctypes.c_char * 8), ("version", ctypes.c_uint32), ("header_bytes", ctypes.c_uint32),
                ("settings", ag2d.WorldSettings), ("counts", ctypes.c_uint32 * 14), ("total", ctypes.c_uint64),
                ("off", ctypes.c_uint64 * SECTIONS), ("len", ctypes.c_uint64 * SECTIONS)]


def _with_colours(blob, word):
    h = _Header.from_buffer_copy(blob[:ctypes.sizeof(_Header)].tobytes())
    assert h.header_bytes == ctypes.sizeof(_Header) and h.len[PREVCOLOR] > 0
    out = blob.copy()
    out[h.off[PREVCOLOR]:h.off[PREVCOLOR] + h.len[PREVCOLOR]].view(np.uint32)[:] = word
    return out


def _dense(n, k):
    side = max(4.0, 1.6 * float(np.sqrt(n)))
    return ag2d.World.from_scene(scenes.make_c1(n, seed=40 + k, width=side, height=side))


@pytest.mark.parametrize("sizes", [(600,), (7000,), (40, 500, 3000)])
def test_clashing_colours_are_dropped(sizes):
    batch = ag2d.Batch([_dense(n, k) for k, n in enumerate(sizes)])
    batch.step(24)
    blob = np.frombuffer(bytes(batch.save()), np.uint8)
    results = []
    for word in (0xFFFFFFFF, 0, 5):   # none; all the first colour; all the sixth
        batch.load(_with_colours(blob, word))
        batch.step(3)
        assert batch.counters()["status"] == 0
        results.append([np.ascontiguousarray(batch.engine.read(f)).view(np.uint8) for f in FIELDS])
    for r in results[1:]:
        for a, b in zip(results[0], r):
            assert np.array_equal(a, b)
