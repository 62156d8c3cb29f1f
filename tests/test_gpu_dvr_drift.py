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


@pytest.mark.parametrize("by", [(90.0001, 0.0), (90.003, 0.0), (179.994, 0.0), (0.0, 89.9995), (90.02, 0.0), (90.06, 0.0)])
@pytest.mark.parametrize("n,air", [(128, False), (121, True)])
def test_cameras_close_to_an_axis_match_plain(n, air, by):
    """Drifts of 1e-6 to 5e-4 cells a sample, on both sides of the rate below which
    the end of a run is looked at."""
    dims, lut = (n, n, n), 64
    views = [dvr.dvr_params(2 * n, 2 * n, _turned(1, by), dims, (1.0, 1.0, 1.0), 0.5, 0.0, lut)]
    vol, table = _volume(dims, 3, air=air), _lut(lut, "cut", 4)
    g = torch.randn((1, 2 * n, 2 * n, 3), generator=torch.Generator("cuda").manual_seed(5), device="cuda")
    a, b = (_run(views, vol, table, g, bricks, True) for bricks in (False, True))
    for k in range(3):
        assert torch.equal(a[k], b[k]), ("image", "transmittance", "workspace")[k]
    assert _close(b[3], a[3]) and _close(b[4], a[4])
