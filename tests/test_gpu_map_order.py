"""Frames of one volume on several streams, with label parameters that change
between them: each frame is the one that its own parameters give.

Streams are kept busy by frames queued before the change, so a frame that does
not wait for the maps of its parameters, or a rebuild that does not wait for the
frames that read the old maps, shows.  The parameters show or hide the whole
volume: a map of the other ones blanks the image."""
import numpy as np
import pytest

from monkeygl_b200 import capi
from monkeygl_b200.camera import Camera
from monkeygl_b200.phantom import make_phantom, make_tf_lut

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

DIMS, SIZE = (128, 120, 136), 384
TF = [(0.0, (0.8, 0.5, 0.4, 0.0)), (0.12, (0.85, 0.55, 0.45, 0.03)), (0.3, (0.9, 0.7, 0.6, 0.12)), (1.0, (1, 1, 0.9, 0.9))]


def _params(shown):
    lp = np.zeros((capi.MAX_LABELS, 3), np.float32)
    lp[:, 1] = 1.0
    lp[:5] = (1.0, 1700.0, 650.0 if shown else 30000.0)
    return lp


@pytest.fixture(scope="module")
def scene():
    ph = make_phantom(DIMS, (0.7, 0.8, 0.9), 5, with_labels=True)
    vol = capi.Volume(ph.volume)
    vol.set_mask(ph.labels)
    for l in range(5):
        vol.set_transfer_function(l, make_tf_lut(TF, 256))
    c = Camera()
    c.anterior()
    c.rotate(25.0, 10.0)
    p = {k: capi.vr_params(SIZE, SIZE, k, c, DIMS, (0.7, 0.8, 0.9)) for k in (capi.RENDER_VR, capi.RENDER_MIP)}
    want = {}
    for shown in (False, True):
        vol.set_label_params(_params(shown))
        for k in p:
            want[k, shown] = vol.render_vr(p[k])
    for k in p:
        assert (want[k, True] != want[k, False]).any()
    return vol, p, want


@pytest.mark.parametrize("kind", [capi.RENDER_VR, capi.RENDER_MIP])
@pytest.mark.parametrize("n_streams", [2, 3, 6])
def test_each_frame_has_its_own_maps(scene, kind, n_streams):
    vol, p, want = scene
    streams = [torch.cuda.Stream() for _ in range(n_streams)]
    frames = []
    shown = False
    for rep in range(12):
        vol.set_label_params(_params(shown))
        # one stream has work ahead of it; another has its frames at once
        order = [streams[(rep + i) % n_streams] for i in range(n_streams)]
        for s, n in [(order[0], 8)] + [(s, 1) for s in order[1:]]:
            for _ in range(n):
                out = torch.zeros((SIZE, SIZE, 3), dtype=torch.uint8, device="cuda")
                s.wait_stream(torch.cuda.current_stream())
                vol.render_vr_device(p[kind], out.data_ptr(), s.cuda_stream)
                frames.append((out, shown, rep))
        shown = not shown
    torch.cuda.synchronize()
    for out, shown, rep in frames:
        assert np.array_equal(out.cpu().numpy(), want[kind, shown]), f"change {rep}, shown: {shown}"


def test_a_host_frame_after_a_change(scene):
    """The image on the host uses the volume's own stream."""
    vol, p, want = scene
    busy = torch.cuda.Stream()
    out = torch.zeros((SIZE, SIZE, 3), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for rep in range(6):
        shown = rep % 2 == 0
        vol.set_label_params(_params(shown))
        for _ in range(6):
            vol.render_vr_device(p[capi.RENDER_VR], out.data_ptr(), busy.cuda_stream)
        assert np.array_equal(vol.render_vr(p[capi.RENDER_VR]), want[capi.RENDER_VR, shown]), f"change {rep}"
    busy.synchronize()
    assert np.array_equal(out.cpu().numpy(), want[capi.RENDER_VR, False])


@pytest.mark.parametrize("change", ["table in place", "table of another length", "table removed", "mask", "mask removed"])
def test_tables_and_masks_change_behind_running_frames(change):
    """Frames queued on a caller's stream keep the table and the mask they were
    queued with; the frame after the change has the new one."""
    ph = make_phantom(DIMS, (0.7, 0.8, 0.9), 5, with_labels=True)
    c = Camera()
    c.anterior()
    c.rotate(25.0, 10.0)
    p = capi.vr_params(SIZE, SIZE, capi.RENDER_VR, c, DIMS, (0.7, 0.8, 0.9))
    other = np.where(ph.labels == 0, 1, 0).astype(np.uint8)

    lut = make_tf_lut(TF, 256)

    def base(vol):
        for l in range(5):
            vol.set_transfer_function(l, lut * np.float32(0.5 if l == 1 else 1.0))
        vol.set_mask(ph.labels)
        vol.set_label_params(_params(True))

    def apply(vol):
        if change == "table in place":
            vol.set_transfer_function(0, lut[::-1])
        elif change == "table of another length":
            vol.set_transfer_function(0, make_tf_lut(TF, 100)[::-1])
        elif change == "table removed":
            vol.set_transfer_function(0, None)
        else:
            vol.set_mask(other if change == "mask" else None)

    vol = capi.Volume(ph.volume)
    base(vol)
    want = [vol.render_vr(p)]
    apply(vol)
    want.append(vol.render_vr(p))
    assert (want[0] != want[1]).any()
    base(vol)
    busy, after = torch.cuda.Stream(), torch.cuda.Stream()
    frames = [torch.zeros((SIZE, SIZE, 3), dtype=torch.uint8, device="cuda") for _ in range(20)]
    torch.cuda.synchronize()
    for f in frames[:-1]:
        vol.render_vr_device(p, f.data_ptr(), busy.cuda_stream)
    apply(vol)
    vol.render_vr_device(p, frames[-1].data_ptr(), after.cuda_stream)
    torch.cuda.synchronize()
    for i, f in enumerate(frames):
        assert np.array_equal(f.cpu().numpy(), want[i == len(frames) - 1]), f"frame {i}"
