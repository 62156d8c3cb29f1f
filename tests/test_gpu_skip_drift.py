"""Leaving out samples (test_gpu_skip.py) with cameras turned in steps.

Nine turns of 10 degrees leave about 3e-8 in the camera matrix where one turn of
90 has 0.  With a pixel pitch of half a voxel, rays that drift by one rounding
cross the face between two bricks; where the labels meet there, the sample
beyond it has another transfer function and another opacity cap.  The image is
that of the march that fetches every sample (MK_VR_NO_SKIP), byte for byte."""
import numpy as np
import pytest

from monkeygl_b200 import capi
from monkeygl_b200.camera import Camera
from monkeygl_b200.phantom import make_tf_lut

pytestmark = pytest.mark.gpu

N = 128
FAINT = [(0.0, (0.9, 0.5, 0.2, 0.02)), (1.0, (0.2, 0.9, 0.9, 0.02))]
PLAIN = [(0.0, (0.8, 0.8, 0.1, 0.3)), (1.0, (0.8, 0.8, 0.1, 0.3))]


def _volume(labels, first, cap):
    """Two labels; the first one hidden (no table) or with its cap soon spent."""
    rng = np.random.default_rng(11)
    vol = capi.Volume(rng.integers(0, 900, (N, N, N)).astype(np.int16))
    vol.set_mask(labels)
    lp = np.zeros((capi.MAX_LABELS, 3), np.float32)
    lp[:, 1] = 1.0
    if first is not None:
        vol.set_transfer_function(1, make_tf_lut(first, 256))
    vol.set_transfer_function(2, make_tf_lut(FAINT, 256))
    lp[1], lp[2] = (cap, 1700.0, 650.0), (1.0, 1700.0, 650.0)
    vol.set_label_params(lp)
    return vol


def _labels(axis, swap):
    """The volume in two halves along `axis`."""
    at = np.arange(N).reshape([-1 if k == 2 - axis else 1 for k in range(3)])
    return np.broadcast_to(np.where((at >= N // 2) != swap, 2, 1), (N, N, N)).astype(np.uint8)


# axis: the one along which the rays drift
@pytest.mark.parametrize("swap", [False, True])
@pytest.mark.parametrize("first,cap", [(None, 1.0), (PLAIN, 0.2)])
@pytest.mark.parametrize("turns,by,axis,invert", [
    (9, (10.0, 0.0), 1, False),
    (27, (10.0, 0.0), 1, False),
    (45, (10.0, 0.0), 1, True),
    (45, (2.0, 0.0), 1, False),
    (18, (10.0, 0.0), 0, False),
    (36, (10.0, 0.0), 0, False),
    (18, (0.0, 10.0), 2, False),
    (36, (0.0, 10.0), 2, True),
    (1, (90.0, 0.0), 1, False),         # drifts below half a rounding: no sample moves
    (1, (180.0, 0.0), 0, False),
])
def test_cameras_turned_in_steps(swap, first, cap, turns, by, axis, invert):
    vol = _volume(_labels(axis, swap), first, cap)
    c = Camera()
    c.anterior()
    for _ in range(turns):
        c.rotate(*by)
    images = {}
    for f in (0, capi.VR_NO_SKIP, capi.VR_NO_COOP, capi.VR_NO_TAIL):
        p = capi.vr_params(2 * N, 2 * N, capi.RENDER_VR, c, (N, N, N), (1.0, 1.0, 1.0), invert_z=invert, flags=f)
        images[f] = vol.render_vr(p)
    want = images[capi.VR_NO_SKIP]
    assert (want != want[0, 0]).any()
    for f, img in images.items():
        assert np.array_equal(img, want), f"flags {f}: {np.count_nonzero(img != want)} bytes differ"


@pytest.mark.parametrize("kind", [capi.RENDER_MIP, capi.RENDER_SURFACE])
@pytest.mark.parametrize("turns,by,axis", [(27, (10.0, 0.0), 1), (18, (0.0, 10.0), 2), (1, (180.0, 0.0), 0)])
def test_cameras_turned_in_steps_mip_and_surface(kind, turns, by, axis):
    vol = _volume(_labels(axis, False), None, 0.0)   # the first label hidden: the labels are looked up
    c = Camera()
    c.anterior()
    for _ in range(turns):
        c.rotate(*by)
    images = [vol.render_vr(capi.vr_params(2 * N, 2 * N, kind, c, (N, N, N), (1.0, 1.0, 1.0), flags=f))
              for f in (0, capi.VR_NO_SKIP)]
    assert np.array_equal(images[0], images[1])


@pytest.mark.parametrize("labelled", [False, True])
@pytest.mark.parametrize("kind", [capi.RENDER_VR, capi.RENDER_MIP, capi.RENDER_SURFACE])
@pytest.mark.parametrize("by", [(90.0001, 0.0), (90.003, 0.0), (179.994, 0.0), (0.0, 89.9995), (90.02, 0.0)])
def test_cameras_close_to_an_axis(labelled, kind, by):
    """Drifts of 2e-6 to 3e-4 voxels a step, on both sides of the rate below which
    an axis is looked at ray by ray (or, without labels, counts as still)."""
    rng = np.random.default_rng(12)
    v = np.full((N, N, N), -900, np.int16)
    v[40:88, 30:100, 24:104] = rng.integers(-300, 1400, (48, 70, 80))
    vol = capi.Volume(v)
    lp = np.zeros((capi.MAX_LABELS, 3), np.float32)
    lp[:, 1] = 1.0
    lp[:3] = (1.0, 1700.0, 650.0)
    if labelled:
        vol.set_mask(_labels(1, False))
        lp[1] = (0.3, 1700.0, 650.0)
    for l in range(3):
        vol.set_transfer_function(l, make_tf_lut(FAINT if l == 2 else PLAIN, 256) *
                                  (np.arange(256) > 90)[:, None].astype(np.float32))
    vol.set_label_params(lp)
    c = Camera()
    c.anterior()
    c.rotate(*by)
    images = [vol.render_vr(capi.vr_params(2 * N, 2 * N, kind, c, (N, N, N), (1.0, 1.0, 1.0), flags=f))
              for f in (0, capi.VR_NO_SKIP)]
    assert (images[1] != images[1][0, 0]).any()
    assert np.array_equal(images[0], images[1]), f"{np.count_nonzero(images[0] != images[1])} bytes differ"
