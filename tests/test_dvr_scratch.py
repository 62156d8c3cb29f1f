"""Scratch of the differentiable renderer: the bytes asked for are those that the
pass uses, and a large one is taken only where it leaves half of the memory."""
import ctypes as C

import pytest

from monkeygl_b200 import dvr
from monkeygl_b200.camera import view_camera

torch = pytest.importorskip("torch")

BRICK = 576 * 16


def _views(n, size, dims, lut, step):
    return [dvr.dvr_params(size, size, view_camera(30.0 + 40.0 * i), dims, (1, 1, 1), step, 1e-4, lut) for i in range(n)]


def _bytes(views, what):
    arr, nv = dvr.view_array(views)
    n = C.c_size_t(0)
    assert dvr._lib().mk_dvr_scratch_bytes(arr, nv, what, C.byref(n)) == 0
    return n.value


@pytest.mark.parametrize("views,size,dims,lut,step,used", [
    (8, 256, (256, 256, 256), 256, 0.5, (1, 1, 1)),
    (1, 128, (192, 192, 192), 16, 0.5, (1, 0, 0)),      # a short table: the backward is plain
    (2, 400, (64, 64, 64), 1024, 0.5, (1, 1, 0)),       # a long one, short rays: so is the LUT-only one
    (1, 321, (211, 190, 157), 1024, 0.5, (1, 0, 0)),    # and few samples per voxel
    (1, 64, (256, 256, 256), 256, 0.5, (0, 0, 0)),      # a small image of a large volume
])
def test_bytes_are_those_of_the_pass(views, size, dims, lut, step, used):
    vs = _views(views, size, dims, lut, step)
    bricks = (dims[0] // 8 + 1) * (dims[1] // 8 + 1) * (dims[2] // 8 + 1)
    got = [_bytes(vs, what) for what in (dvr._FORWARD, dvr._BACKWARD, dvr._BACKWARD_LUT)]
    assert tuple(int(b > 0) for b in got) == used
    for b, quads in zip(got, (1, 2, 1)):
        assert b == 0 or quads * bricks * BRICK <= b < quads * bricks * BRICK + 32 * bricks + (1 << 17)


def test_large_scratch_leaves_half_of_the_memory(monkeypatch):
    vs = _views(4, 512, (512, 512, 512), 256, 0.5)
    arr, nv = dvr.view_array(vs)
    need = _bytes(vs, dvr._BACKWARD)
    assert need > dvr._LARGE_SCRATCH
    asked = []
    state = dict(free=0, reserved=0, allocated=0, capturing=False)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state["capturing"])
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device=None: (state["free"], 180 << 30))
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda device=None: state["reserved"])
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda device=None: state["allocated"])
    monkeypatch.setattr(torch, "empty", lambda n, **kw: asked.append(n) or "scratch")

    def take(**kw):
        state.update(dict(free=0, reserved=0, allocated=0, capturing=False), **kw)
        asked.clear()
        r = dvr._scratch(arr, nv, dvr._BACKWARD, "cuda:0")
        assert r == (("scratch", need) if asked else (None, 0))
        return bool(asked)

    assert take(free=2 * need)
    assert not take(free=2 * need - 2)
    assert take(free=need, reserved=3 * need, allocated=2 * need)
    assert not take(free=need, reserved=3 * need, allocated=3 * need)
    assert take(free=0, capturing=True)         # no query of the device while a graph is recorded
