"""Host memory that is page-locked in part only, or for reading only: refused or copied, never reached by a kernel beyond
its registration. The engine works on after a refusal.
"""
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ag2d = pytest.importorskip("ag2d")
torch = pytest.importorskip("torch")
from ag2d import scenes  # noqa: E402

PAGE = 4096


@pytest.fixture()
def registered():
    """Arrays of 64 pages of which the first ones are page-locked: registered(pages, flags)."""
    rt, held = torch.cuda.cudart(), []

    def make(pages, flags=0):
        a = np.frombuffer(mmap.mmap(-1, 64 * PAGE), np.uint8)
        assert int(rt.cudaHostRegister(a.ctypes.data, pages * PAGE, flags)) == 0
        held.append(a)
        return a

    torch.cuda.init()
    yield make
    for a in held:
        assert int(rt.cudaHostUnregister(a.ctypes.data)) == 0


def _world():
    w = ag2d.World.from_scene(scenes.make_c1(600, seed=1, width=60.0, height=30.0))
    w.step(3)
    return w


@pytest.mark.parametrize("field,bytes_each", [(ag2d.BODY_POSE, 12), (ag2d.BODY_VEL_X, 4), (ag2d.BODY_STATE, 4),
                                              (ag2d.BODY_SLEEP_TIMER, 4)])
def test_reads(registered, field, bytes_each):
    w = _world()
    nb, _ = w.counts()
    size = nb * bytes_each
    want = np.ascontiguousarray(w.read(field)).view(np.uint8).reshape(-1)
    whole = registered(64)
    assert w.read(field, whole[:size]).view(np.uint8).reshape(-1).tobytes() == want.tobytes()
    odd = registered(64)   # from inside a registration to its last byte
    assert w.read(field, odd[-size:]).view(np.uint8).reshape(-1).tobytes() == want.tobytes()
    part = registered(2)
    for at in (2 * PAGE - 4, 2 * PAGE - size + 4):   # only the first, all but the last four bytes
        with pytest.raises(ag2d.Ag2dError):
            w.read(field, part[at:at + size])
        with pytest.raises(ag2d.Ag2dError):
            w.read_async(field, part[at:at + size])
    assert not part.any()
    assert w.read(field, part[2 * PAGE:2 * PAGE + size]).view(np.uint8).reshape(-1).tobytes() == want.tobytes()
    w.step(1)
    assert w.counters()["status"] == 0


def test_checkpoints(registered):
    batch = ag2d.Batch([_world()])
    saved = np.array(batch.save())
    assert saved.size < 60 * PAGE
    pose = batch.engine.read(ag2d.BODY_POSE).tobytes()
    part = registered(4)
    part[:saved.size] = saved
    with pytest.raises(ag2d.Ag2dError):
        batch.load(part[:saved.size])
    for blob in (registered(64), registered(64, 8)):   # 8: cudaHostRegisterReadOnly
        blob[:saved.size] = saved
        batch.step(2)
        batch.load(blob[:saved.size])
        assert batch.engine.read(ag2d.BODY_POSE).tobytes() == pose
