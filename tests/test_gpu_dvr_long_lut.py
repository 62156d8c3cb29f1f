"""Gradients of the bricked differentiable renderer over the lengths of its table
where the window of LUT sums and the use of bricks change (256, 512, 750 entries):
as the plain calls, up to the order of the sums (4e-5 in the 2-norm)."""
import pytest

from test_gpu_dvr_bricks import _close, _lut, _run, _views, _volume, torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["cut", "seen"])
@pytest.mark.parametrize("lut", [256, 257, 512, 513, 750, 751, 1024])
@pytest.mark.parametrize("dims,size,views,step", [((40, 31, 50), (65, 47), 2, 0.12), ((48, 56, 64), (400, 380), 2, 0.3)])
def test_tables_of_all_lengths(dims, size, views, step, lut, kind):
    vol, table = _volume(dims, 3), _lut(lut, kind, 4)
    vs = _views(views, *size, dims, lut, step, 1e-4)
    g = torch.randn((views, size[1], size[0], 3), generator=torch.Generator("cuda").manual_seed(5), device="cuda")
    for volgrad in (True, False):
        a, b = (_run(vs, vol, table, g, bricks, volgrad) for bricks in (False, True))
        for k in range(3):
            assert torch.equal(a[k], b[k])
        assert _close(b[3], a[3])
        if volgrad:
            assert _close(b[4], a[4])
