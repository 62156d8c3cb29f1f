"""The differentiable renderer over bricks (the *_scratch calls with scratch)
against the plain calls on the same inputs: image, transmittance, sample
counts and checkpoints bit for bit, gradients up to the order of their sums.

Sizes sit at the edges of the 8^3 bricks (dims 1, 7, 8, 9, 17), of the 16x8
pixel blocks, and on both sides of the ray count that picks the forward
kernel's look-ahead.  Transfer functions: transparent below a cut (bricks left
out), opaque entries (a division by 1 - a = 0), everything visible.  A
gradient is a sum of up to about 1e5 fp32 terms added in another order, each
sum with a relative rounding of about sqrt(1e5) * 6e-8 = 2e-5; asserted at
twice that in the 2-norm."""
import ctypes as C

import numpy as np
import pytest

from monkeygl_b200 import dvr
from monkeygl_b200.camera import Camera

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _ptr(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


def _volume(dims, seed, air=True):
    """Values with padding (exactly equal voxels), noise and dense spots."""
    x, y, z = dims
    g = torch.Generator("cuda").manual_seed(seed)
    v = 0.25 + 0.01 * torch.randn((z, y, x), generator=g, device="cuda")
    v += 0.6 * (torch.rand((z, y, x), generator=g, device="cuda") > 0.995)
    if air:
        v[: z // 3] = 0.0
        v[:, :, : x // 4] = 0.0
    return v.clamp_(0.0, 1.0).contiguous()


def _lut(n, kind, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    l = rng.uniform(0.1, 1.0, (n, 4)).astype(np.float32)
    t = np.arange(n) / max(1, n - 1)
    l[:, 3] = {"cut": np.clip(t - 0.35, 0, 1), "seen": 0.002 + 0.3 * t ** 2, "opaque": np.where(t > 0.5, 1.0, 0.0)}[kind]
    return torch.tensor(l, device="cuda")


def _views(n, w, h, dims, lut, step, t_min):
    out = []
    for i in range(n):
        c = Camera()
        c.anterior()
        c.rotate(20.0 + 97.0 * i, 15.0 * (i % 3))
        out.append(dvr.dvr_params(w, h, c, dims, (1.0, 0.9, 1.1), step, t_min, lut))
    return out


def _run(views, vol, lut, g, bricks, volgrad):
    L = dvr._lib()
    arr, nv = dvr.view_array(views)
    p = arr[0]
    images = torch.empty((nv, p.height, p.width, 3), device="cuda")
    trans = torch.empty((nv, p.height, p.width), device="cuda")
    work = torch.full((dvr.workspace_floats(arr),), -7.0, device="cuda")
    g_lut = torch.zeros_like(lut)
    g_vol = torch.zeros_like(vol) if volgrad else None
    n = C.c_size_t(0)
    assert L.mk_dvr_scratch_bytes(arr, nv, int(volgrad), C.byref(n)) == 0
    assert n.value > 0
    scratch = torch.full((n.value,), 0xA5, dtype=torch.uint8, device="cuda") if bricks else None
    size = n.value if bricks else 0
    assert L.mk_dvr_forward_scratch(arr, nv, _ptr(vol), _ptr(lut), _ptr(images), _ptr(trans), _ptr(work),
                                    _ptr(scratch), size, None) == 0
    assert L.mk_dvr_backward_scratch(arr, nv, _ptr(vol), _ptr(lut), _ptr(work), _ptr(g), _ptr(g_lut), _ptr(g_vol),
                                     _ptr(scratch), size, None) == 0
    torch.cuda.synchronize()
    return images, trans, work, g_lut, g_vol


def _close(a, b):
    return (a - b).norm().item() <= 4e-5 * b.norm().item()


@pytest.mark.parametrize("dims,size,views,lut,kind,step,t_min", [
    ((9, 8, 17), (20, 12), 1, 64, "cut", 0.02, 1e-4),
    ((7, 7, 7), (9, 7), 2, 64, "seen", 0.02, 0.0),
    ((1, 24, 33), (31, 17), 3, 64, "seen", 0.004, 0.0),
    ((40, 31, 50), (65, 47), 4, 256, "cut", 0.12, 1e-4),
    ((40, 31, 50), (65, 47), 2, 256, "opaque", 0.13, 0.0),
    ((64, 64, 64), (110, 105), 33, 1000, "cut", 1.0, 0.05),
    ((48, 56, 64), (400, 380), 2, 2, "seen", 0.3, 1e-3),
    ((32, 32, 32), (24, 24), 1, 100, "cut", 0.1, 2.0),
    ((170, 165, 168), (160, 150), 1, 64, "cut", 0.5, 1e-3),
])
def test_bricks_match_plain(dims, size, views, lut, kind, step, t_min):
    vol, table = _volume(dims, 3), _lut(lut, kind, 4)
    vs = _views(views, *size, dims, lut, step, t_min)
    g = torch.randn((views, size[1], size[0], 3), generator=torch.Generator("cuda").manual_seed(5), device="cuda")
    for volgrad in (True, False):
        a, b = (_run(vs, vol, table, g, bricks, volgrad) for bricks in (False, True))
        for k in range(3):
            assert torch.equal(a[k], b[k]), ("image", "transmittance", "workspace")[k]
        assert torch.isfinite(a[3]).all()
        assert _close(b[3], a[3])
        if volgrad:
            assert _close(b[4], a[4])


def test_gradients_that_are_not_finite_spread_as_before():
    dims, n = (40, 31, 50), 64
    vol, table = _volume(dims, 6), _lut(n, "cut", 7)
    vs = _views(2, 33, 29, dims, n, 0.12, 1e-4)
    g = torch.randn((2, 29, 33, 3), generator=torch.Generator("cuda").manual_seed(8), device="cuda")
    g[0, 14, 16, 1] = float("inf")
    g[1, 10, 12, 0] = float("nan")
    a, b = (_run(vs, vol, table, g, bricks, True) for bricks in (False, True))
    for k in (3, 4):
        fine = torch.isfinite(a[k])
        assert torch.equal(fine, torch.isfinite(b[k])) and not fine.all()
        assert _close(b[k][fine], a[k][fine])


def test_values_outside_the_unit_range():
    """Voxels beyond what the range test of a brick can place (and NaN) are
    rendered, not left out."""
    dims, n = (24, 24, 24), 64
    vol, table = _volume(dims, 9), _lut(n, "cut", 10)
    vol[5, 5, 5], vol[12, 12, 12], vol[18, 9, 9] = 1e30, float("nan"), -50.0
    vs = _views(1, 40, 40, dims, n, 0.08, 0.0)
    g = torch.ones((1, 40, 40, 3), device="cuda")
    a, b = (_run(vs, vol, table, g, bricks, True) for bricks in (False, True))
    assert torch.equal(a[0], b[0]) and torch.equal(a[2], b[2])
    for k in (3, 4):
        fine = torch.isfinite(a[k])
        assert torch.equal(fine, torch.isfinite(b[k]))
        assert _close(b[k][fine], a[k][fine])
