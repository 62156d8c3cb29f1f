"""Leaving out samples that cannot change a pixel (distance map, busy map, MIP
bounds) gives the image of the march that fetches every sample
(MK_VR_NO_SKIP), byte for byte, with and without the cooperative rounds and the
hand-off launch.

The volumes have sides around multiples of the brick (8) and of the tile, noise,
padding and labelled objects; the transfer functions reach from mostly
transparent to soft tissue visible under spent opacity caps, hidden labels and
more capped labels than the shared accumulators hold."""
import numpy as np
import pytest

from monkeygl_b200 import capi
from monkeygl_b200.camera import Camera
from monkeygl_b200.phantom import make_phantom, make_tf_lut

pytestmark = pytest.mark.gpu

SPARSE = [(0.0, (0.7, 0.3, 0.2, 0.0)), (0.25, (0.8, 0.4, 0.3, 0.0)), (0.5, (0.9, 0.7, 0.5, 0.4)), (1.0, (1, 1, 1, 0.9))]
DENSE = [(0.0, (0.8, 0.5, 0.4, 0.0)), (0.12, (0.85, 0.55, 0.45, 0.03)), (0.3, (0.9, 0.7, 0.6, 0.12)), (1.0, (1, 1, 0.9, 0.9))]
OPAQUE = [(0.0, (0.8, 0.5, 0.4, 0.05)), (0.2, (0.85, 0.55, 0.45, 1.0)), (1.0, (1, 1, 0.9, 1.0))]


def _volume(dims, tf, caps, labels, seed, lut_len=256):
    ph = make_phantom(dims, (0.7, 0.8, 0.9), seed, with_labels=True)
    lab = ph.labels.copy()
    if labels > 5:                      # slabs of further labels inside the body
        z = np.arange(dims[2]) * labels // dims[2]
        body = ph.volume > -500
        lab = np.where(body & (lab == 0), z[:, None, None].astype(np.uint8), lab)
    vol = capi.Volume(ph.volume)
    vol.set_mask(lab)
    lp = np.zeros((capi.MAX_LABELS, 3), np.float32)
    lp[:, 1] = 1.0
    rng = np.random.default_rng(seed)
    for l in range(labels):
        vol.set_transfer_function(l, make_tf_lut(tf, lut_len))
        lp[l] = (caps if l == 0 else float(rng.uniform(0.3, 1.0)), 1700.0, 650.0)
    if labels == 5:
        lp[2, 0] = 0.0                  # a hidden object still steers the step
    vol.set_label_params(lp)
    return vol


@pytest.mark.parametrize("dims,size,tf,caps,labels,kind,turn,zoom,invert,crop", [
    ((64, 64, 48), (96, 80), DENSE, 0.4, 5, capi.RENDER_VR, (20, 10), 1.0, False, False),
    ((65, 71, 57), (131, 77), DENSE, 0.2, 5, capi.RENDER_VR, (75, -30), 1.4, True, True),
    ((128, 96, 130), (200, 190), SPARSE, 0.4, 5, capi.RENDER_VR, (140, 0), 0.8, False, False),
    ((40, 48, 200), (64, 160), SPARSE, 1.0, 5, capi.RENDER_VR, (0, 0), 1.0, False, True),
    ((63, 64, 65), (70, 70), DENSE, 0.5, 24, capi.RENDER_VR, (33, 5), 1.2, False, False),
    ((64, 64, 64), (90, 64), OPAQUE, 0.3, 5, capi.RENDER_VR, (10, 40), 1.0, False, False),
    ((9, 7, 8), (33, 21), DENSE, 0.3, 5, capi.RENDER_VR, (45, 45), 1.0, False, False),
    ((65, 71, 57), (131, 77), SPARSE, 0.4, 5, capi.RENDER_MIP, (75, -30), 1.4, True, True),
    ((128, 96, 130), (200, 190), SPARSE, 0.4, 5, capi.RENDER_MIP, (140, 0), 0.8, False, False),
    ((9, 7, 8), (33, 21), SPARSE, 1.0, 5, capi.RENDER_MIP, (45, 45), 1.0, False, False),
    ((65, 71, 57), (131, 77), SPARSE, 0.4, 5, capi.RENDER_MIP, (15, 30), 1.0, False, "wide"),
    ((65, 71, 57), (131, 77), DENSE, 0.4, 5, capi.RENDER_VR, (15, 30), 1.0, False, "wide"),
    ((64, 64, 64), (90, 64), SPARSE, 0.4, 5, capi.RENDER_MIP, (10, 40), 2e-6, False, False),
    ((64, 64, 64), (90, 64), SPARSE, 0.4, 5, capi.RENDER_MIP, (10, 40), 30.0, False, False),
    ((65, 71, 57), (131, 77), SPARSE, 0.4, 5, capi.RENDER_SURFACE, (75, -30), 1.4, True, True),
])
def test_skipping_leaves_the_image(dims, size, tf, caps, labels, kind, turn, zoom, invert, crop):
    vol = _volume(dims, tf, caps, labels, 3)
    if kind == capi.RENDER_MIP:
        lp = np.zeros((capi.MAX_LABELS, 3), np.float32)
        lp[:labels] = (1.0, 1700.0, 650.0)          # every label visible, one window
        lp[labels:, 1] = 1.0
        vol.set_label_params(lp)
    c = Camera()
    c.anterior()
    c.rotate(*turn)
    c.zoom(zoom)
    c.pan(3.0, -5.0)
    wide = (-3, dims[0] + 4, 0, dims[1], -1, dims[2] + 2)
    voi = wide if crop == "wide" else (dims[0] // 5, dims[0] - 3, 2, dims[1] * 3 // 4, dims[2] // 7, dims[2] - 2) if crop else None
    images = {}
    flags = [0, capi.VR_NO_SKIP]
    if kind == capi.RENDER_VR:
        flags += [capi.VR_NO_COOP, capi.VR_NO_TAIL, capi.VR_NO_SKIP | capi.VR_NO_COOP]
    for f in flags:
        p = capi.vr_params(*size, kind, c, dims, (0.7, 0.8, 0.9), invert_z=invert, voi=voi, flags=f,
                           background=(0.1, 0.2, 0.3, 1.0))
        images[f] = vol.render_vr(p)
    want = images[capi.VR_NO_SKIP]
    if zoom > 1e-3:                     # (else the volume is less than a pixel)
        assert (want != want[0, 0]).any()
    for f, img in images.items():
        assert np.array_equal(img, want), f"flags {f}: {np.count_nonzero(img != want)} bytes differ"
