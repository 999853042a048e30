"""Reads into pageable memory give the same bytes as reads into page-locked memory, the first and later ones, for packed
fields, fields copied as they lie and the phase taps, in worlds of 200 to 400,000 bodies.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ag2d = pytest.importorskip("ag2d")
from ag2d import scenes  # noqa: E402


@pytest.mark.parametrize("n", [200, 30_000, 400_000])
def test_pageable_reads_equal_page_locked_ones(n):
    side = 3.0 * float(np.sqrt(n))
    w = ag2d.World.from_scene(scenes.make_c3(n, 5, extent=side))
    w.run_phase(ag2d.PHASE_COLLIDE)
    for f in (ag2d.MANIFOLDS, ag2d.PAIRS, ag2d.DYN_SORTED, ag2d.BODY_POSE, ag2d.BODY_VEL_X, ag2d.BODY_SLEEP_TIMER):
        first = w.read(f).tobytes()
        assert first
        out = ag2d.host_empty(len(first))
        assert w.read(f, out).tobytes() == first
        assert w.read(f).tobytes() == first
