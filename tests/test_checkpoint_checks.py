"""A checkpoint whose sections are not those of its counts is refused before anything is allocated or launched, and one
whose sections lie elsewhere than a save puts them loads as before.
"""
import ctypes
import os

import numpy as np
import pytest

ag2d = pytest.importorskip("ag2d")
from ag2d import scenes  # noqa: E402

SECTIONS = 29
COUNTS = ("worlds", "bodies", "colliders", "circles", "boxes", "polygons", "poly_verts", "materials", "prev", "static",
          "last_manifolds", "isle", "last_pairs", "pad")


class Header(ctypes.Structure):
    _fields_ = [("magic", ctypes.c_char * 8), ("version", ctypes.c_uint32), ("header_bytes", ctypes.c_uint32),
                ("settings", ag2d.WorldSettings), ("counts", ctypes.c_uint32 * len(COUNTS)), ("total", ctypes.c_uint64),
                ("off", ctypes.c_uint64 * SECTIONS), ("len", ctypes.c_uint64 * SECTIONS)]


def _lengths(n):
    b, c, wp = n["bodies"], n["colliders"], n["worlds"] + 1
    return [16 * b, 16 * b, 8 * b, 4 * b, 4 * b, 4 * b, b, 4 * b, 4 * c, 4 * c, 4 * c, 16 * c, 16 * c, 16 * c, 4 * c, 4 * c,
            4 * n["circles"], 8 * n["boxes"], 4 * n["polygons"], 4 * n["polygons"], 8 * n["poly_verts"],
            8 * n["poly_verts"], 16 * n["materials"], 64 * n["prev"], 4 * n["prev"], 4 * wp, 4 * wp, 64 * n["isle"],
            4 * n["isle"]]


def _blob(edit=None):
    n = dict.fromkeys(COUNTS, 0)
    n.update(worlds=1, bodies=3, colliders=5, circles=2, boxes=2, polygons=1, poly_verts=4, materials=2, prev=2, isle=1)
    h = Header(magic=b"AG2DCKPT", version=3, header_bytes=ctypes.sizeof(Header))
    h.settings = ag2d.WorldSettings(dt=1.0 / 60.0, velocity_iterations=8, position_iterations=3, angular_damping=1.0)
    at = (ctypes.sizeof(Header) + 255) & ~255
    for k, length in enumerate(_lengths(n)):
        h.off[k], h.len[k] = at, length
        at += (length + 255) & ~255
    h.total = at
    h.counts[:] = [n[k] for k in COUNTS]
    if edit:
        edit(h)
    return bytes(h) + bytes(at + 4096 - ctypes.sizeof(Header))


def _restore(blob):
    out = ctypes.c_void_p()
    return ag2d.lib.ag2d_batch_restore(blob, len(blob), 0, ctypes.byref(out))


def _grow(k, by):
    def edit(h):
        h.len[k] += by
        h.total += 1024
    return edit


@pytest.mark.parametrize("by", [-1, 1, 16])
@pytest.mark.parametrize("section", range(SECTIONS))
def test_a_section_of_another_size_is_refused(section, by):
    assert _restore(_blob(_grow(section, by))) == ag2d.ERR_INVALID_ARG


@pytest.mark.skipif(os.path.exists("/dev/nvidiactl"), reason="would be restored where there is a device")
def test_the_sizes_of_the_counts_are_accepted():
    assert _restore(_blob()) == ag2d.ERR_NO_DEVICE


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [4, 16])
def test_sections_at_other_offsets_load(shift):
    batch = ag2d.Batch([ag2d.World.from_scene(scenes.make_c1(64, seed=k, width=12.0, height=12.0)) for k in range(2)])
    batch.step(30)
    saved = batch.save()
    h = Header.from_buffer_copy(saved[:ctypes.sizeof(Header)].tobytes())
    moved = ag2d.host_empty(saved.size + 1024 * SECTIONS)
    moved[:] = 0
    assert moved.size <= 1 << 20   # the size that one kernel reads over the link
    at = (ctypes.sizeof(Header) + 255) & ~255
    for k in range(SECTIONS):
        at += shift
        moved[at:at + h.len[k]] = saved[h.off[k]:h.off[k] + h.len[k]]
        h.off[k] = at
        at += (h.len[k] + 255) & ~255
    h.total = at
    moved[:ctypes.sizeof(Header)] = np.frombuffer(bytes(h), np.uint8)
    states = []
    for blob in (saved, moved):
        batch.load(blob)
        batch.step(5)
        states.append([batch.engine.read(f).view(np.uint32) for f in
                       (ag2d.BODY_POSE, ag2d.BODY_VEL_X, ag2d.BODY_VEL_Y, ag2d.BODY_STATE)])
    for a, b in zip(*states):
        assert np.array_equal(a, b)
