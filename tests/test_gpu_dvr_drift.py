"""The bricked differentiable renderer with cameras turned in steps.

Nine turns of 10 degrees leave about 3e-8 in the camera matrix where one turn of
90 has 0, so rays that should run along a plane drift by one rounding.  With a
pixel pitch of half a voxel whole columns of rays lie on the faces of the 8^3
bricks and cross them by that drift.  Image, transmittance and workspace equal
the plain calls' bit for bit; gradients to 4e-5 in the 2-norm (their sums' order,
as for the other views)."""
import pytest

from monkeygl_b200 import dvr
from monkeygl_b200.camera import Camera

from test_gpu_dvr_bricks import _close, _lut, _run, _volume, torch

pytestmark = pytest.mark.gpu


def _turned(turns, by):
    c = Camera()
    c.anterior()
    for _ in range(turns):
        c.rotate(*by)
    return c


@pytest.mark.parametrize("n,turns,by", [
    (128, 9, (10.0, 0.0)),
    (128, 27, (10.0, 0.0)),
    (128, 18, (10.0, 0.0)),
    (128, 9, (0.0, 10.0)),
    (256, 9, (10.0, 0.0)),
    (256, 6, (15.0, 0.0)),
    (256, 18, (5.0, 0.0)),
    (120, 9, (10.0, 0.0)),      # the volume's own faces are no brick faces
    (128, 1, (90.0, 0.0)),      # a drift below half a rounding: no sample moves
    (128, 1, (180.0, 0.0)),
])
def test_cameras_turned_in_steps_match_plain(n, turns, by):
    dims, lut = (n, n, n), 64
    views = [dvr.dvr_params(2 * n, 2 * n, _turned(turns, by), dims, (1.0, 1.0, 1.0), 0.5, 0.0, lut)]
    vol, table = _volume(dims, 3, air=False), _lut(lut, "cut", 4)
    g = torch.randn((1, 2 * n, 2 * n, 3), generator=torch.Generator("cuda").manual_seed(5), device="cuda")
    a, b = (_run(views, vol, table, g, bricks, True) for bricks in (False, True))
    for k in range(3):
        assert torch.equal(a[k], b[k]), ("image", "transmittance", "workspace")[k]
    assert _close(b[3], a[3]) and _close(b[4], a[4])
