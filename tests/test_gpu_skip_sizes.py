"""Leaving out samples (test_gpu_skip.py) at the sizes where the maps are built
another way: more than 4096 slices (every empty brick its own step, no runs on step
L1/8), the last size with long runs, more than 8192 bricks (the distances of a
slice in one block), slices above 48 KB of shared memory and above what a block can
have."""
import numpy as np
import pytest

from monkeygl_b200 import capi
from monkeygl_b200.camera import Camera
from monkeygl_b200.phantom import make_tf_lut

from test_gpu_skip import DENSE, SPARSE

pytestmark = pytest.mark.gpu


def _volume(dims, tf, seed):
    """Air, a body in the middle third along every axis with noise, two labels,
    dense specks."""
    x, y, z = dims
    rng = np.random.default_rng(seed)
    v = np.full((z, y, x), -1000, np.int16)
    lab = np.zeros((z, y, x), np.uint8)
    body = tuple(slice(n // 4, max(n // 4 + 1, 3 * n // 4)) for n in (z, y, x))
    shape = v[body].shape
    v[body] = rng.integers(0, 80, shape, dtype=np.int16)
    v[body][rng.random(shape) > 0.999] = 1200
    lab[body][: shape[0] // 2] = 1
    lab[body][:, : shape[1] // 3] = 2
    vol = capi.Volume(v)
    vol.set_mask(lab)
    lp = np.zeros((capi.MAX_LABELS, 3), np.float32)
    lp[:, 1] = 1.0
    for l, cap in ((0, 0.4), (1, 0.3), (2, 0.7)):
        vol.set_transfer_function(l, make_tf_lut(tf, 256))
        lp[l] = (cap, 1700.0, 650.0)
    vol.set_label_params(lp)
    return vol


@pytest.mark.parametrize("dims,spacing,tf", [
    ((16, 16, 4200), (4.0, 4.0, 0.05), DENSE),
    ((16, 16, 4200), (4.0, 4.0, 0.05), SPARSE),
    ((24, 24, 4096), (4.0, 4.0, 0.05), DENSE),
    ((24, 24, 4096), (4.0, 4.0, 0.05), SPARSE),
    ((170, 165, 168), (0.7, 0.7, 0.7), DENSE),
    ((170, 165, 168), (0.7, 0.7, 0.7), SPARSE),
    # (nine slices make steps that miss the specks, all that SPARSE shows)
    ((1264, 1270, 9), (0.3, 0.3, 10.0), DENSE),
    ((2568, 2570, 9), (0.3, 0.3, 20.0), DENSE),
])
@pytest.mark.parametrize("turn", [(20, 10), (0, 90)], ids=["turned", "along"])
def test_skipping_leaves_the_image(dims, spacing, tf, turn):
    vol = _volume(dims, tf, 3)
    c = Camera()
    c.anterior()
    c.rotate(*turn)
    images = {}
    for f in (0, capi.VR_NO_SKIP, capi.VR_NO_COOP, capi.VR_NO_TAIL):
        p = capi.vr_params(150, 130, capi.RENDER_VR, c, dims, spacing, flags=f, background=(0.1, 0.2, 0.3, 1.0))
        images[f] = vol.render_vr(p)
    want = images[capi.VR_NO_SKIP]
    assert (want != want[0, 0]).any()
    for f, img in images.items():
        assert np.array_equal(img, want), f"flags {f}: {np.count_nonzero(img != want)} bytes differ"
