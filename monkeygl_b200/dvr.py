"""Differentiable volume rendering on the sm_100a kernels (mk_dvr_* in
include/monkeygl_b200.h), exposed as a torch.autograd.Function.

    views = [dvr_params(256, 256, view_camera(a), dims, spacing) for a in angles]
    images = render(volume, lut, views)          # (V, H, W, 3), differentiable
    loss = ((images - target) ** 2).mean()
    loss.backward()                              # volume.grad, lut.grad

`volume` is a float32 CUDA tensor (dim_z, dim_y, dim_x) with values in [0, 1]
and `lut` a float32 CUDA tensor (n, 4) of RGBA entries.  Torch provides the
device memory and the stream; forward and backward are the library's kernels.
The method (fixed step, exact trilinear, value as LUT coordinate,
front-to-back compositing with termination at t_min) is described in
monkeygl_b200/csrc/mk_dvr.cu.
"""
from __future__ import annotations

import ctypes as C

from . import capi
from .capi import DVRParams
from .camera import volume_factors


def _lib():
    return capi.lib()


def dvr_params(width, height, camera, dims, spacing, step_voxels=0.5, t_min=1e-4, lut_len=256) -> DVRParams:
    """Parameters of one view.  The step is in voxels of the longest axis:
    MonkeyGL's ray parameter advances by 1/dim_z per voxel (core/kernel.cu:169)."""
    mls, _ = volume_factors(dims, spacing)
    p = DVRParams()
    p.width, p.height = int(width), int(height)
    for k in range(3):
        p.dims[k] = int(dims[k])
        p.max_len_spacing[k] = mls[k]
    for i, m in enumerate(camera.flat()):
        p.transform[i] = m
    p.scale = float(camera.scale)
    p.x_translate = float(camera.x_translate)
    p.y_translate = float(camera.y_translate)
    p.step = float(step_voxels) / float(dims[2])
    p.t_min = float(t_min)
    p.lut_len = int(lut_len)
    return p


def params_flat(p: DVRParams):
    """The parameter block of oracle.mko_dvr_forward_d (FP64 restatement)."""
    import numpy as np
    return np.array([p.width, p.height, *p.dims, *p.max_len_spacing, *p.transform, p.scale, p.x_translate,
                     p.y_translate, p.step, p.t_min, p.lut_len], np.float64)


def _check(rc, where):
    if rc != 0:
        raise capi.MonkeyGLError(rc, where, capi.lib().mk_last_error().decode(errors="replace"))


def _ptr(t):
    return t.data_ptr() if t is not None else None


def view_array(views):
    """The views as a C array of DVRParams (ctypes)."""
    if not isinstance(views, list):
        views = list(views)
    return (DVRParams * len(views))(*views), len(views)


def workspace_floats(views) -> int:
    arr, n = view_array(views)
    out = C.c_size_t(0)
    _check(_lib().mk_dvr_workspace_floats(arr, n, C.byref(out)), "mk_dvr_workspace_floats")
    return out.value


# The pass that scratch is for (mk_dvr_scratch_bytes).
_FORWARD, _BACKWARD, _BACKWARD_LUT = 0, 1, 2
_LARGE_SCRATCH = 2 << 30


def _scratch(arr, nv, what, device):
    """Scratch for one call on the current stream (which the caching allocator
    hands the memory back to), or none.  It takes 18 or 36 bytes a voxel, so a large
    one is only asked for if it leaves half of the memory there is to have: the
    program around keeps room, and an allocation that would fail does not make
    torch empty its cache on every call."""
    import torch
    n = C.c_size_t(0)
    _check(_lib().mk_dvr_scratch_bytes(arr, nv, what, C.byref(n)), "mk_dvr_scratch_bytes")
    if n.value == 0:
        return None, 0
    if n.value >= _LARGE_SCRATCH and not torch.cuda.is_current_stream_capturing():
        room = torch.cuda.mem_get_info(device)[0] + torch.cuda.memory_reserved(device) - torch.cuda.memory_allocated(device)
        if n.value > room // 2:
            return None, 0
    try:
        return torch.empty(n.value, dtype=torch.uint8, device=device), n.value
    except torch.cuda.OutOfMemoryError:
        return None, 0


def _torch_function():
    import torch

    class VolumeRender(torch.autograd.Function):
        @staticmethod
        def forward(ctx, volume, lut, views):
            if not (volume.is_cuda and lut.is_cuda):
                raise ValueError("volume and lut must be CUDA tensors")
            volume = volume.detach().contiguous().float()
            lut = lut.detach().contiguous().float()
            L = _lib()
            arr, nv = view_array(views)
            p0 = arr[0]
            if p0.lut_len != lut.shape[0] or tuple(p0.dims) != tuple(volume.shape[::-1]):
                raise ValueError("view parameters do not match the volume or LUT")
            # the other views share the first one's size, dims and LUT length
            # (compared as bytes: a ctypes field costs more than a small launch)
            raw, n = memoryview(arr).cast("B"), C.sizeof(DVRParams)
            for o in range(n, len(raw), n):
                if raw[o + 8:o + 20] != raw[8:20] or raw[o + n - 4:o + n] != raw[n - 4:n]:
                    raise ValueError("view parameters do not match the volume or LUT")
                if raw[o:o + 8] != raw[:8]:
                    raise ValueError("the views of one render must share width and height")
            stream = torch.cuda.current_stream(volume.device).cuda_stream
            images = torch.empty((nv, p0.height, p0.width, 3), dtype=torch.float32, device=volume.device)
            trans = torch.empty((nv, p0.height, p0.width), dtype=torch.float32, device=volume.device)
            work = None
            if ctx.needs_input_grad[0] or ctx.needs_input_grad[1]:
                work = torch.empty(workspace_floats(arr), dtype=torch.float32, device=volume.device)
            tmp, tmp_bytes = _scratch(arr, nv, _FORWARD, volume.device)
            _check(L.mk_dvr_forward_scratch(arr, nv, _ptr(volume), _ptr(lut), _ptr(images), _ptr(trans), _ptr(work),
                                            _ptr(tmp), tmp_bytes, stream), "mk_dvr_forward")
            ctx.views = arr
            ctx.work = work
            ctx.save_for_backward(volume, lut)
            return images

        @staticmethod
        def backward(ctx, grad_images):
            volume, lut = ctx.saved_tensors
            L = _lib()
            stream = torch.cuda.current_stream(volume.device).cuda_stream
            grad_lut = torch.zeros_like(lut)
            grad_vol = torch.zeros_like(volume) if ctx.needs_input_grad[0] else None
            g = grad_images.contiguous().float()
            what = _BACKWARD_LUT if grad_vol is None else _BACKWARD
            tmp, tmp_bytes = _scratch(ctx.views, len(ctx.views), what, volume.device)
            _check(L.mk_dvr_backward_scratch(ctx.views, len(ctx.views), _ptr(volume), _ptr(lut), _ptr(ctx.work), _ptr(g),
                                             _ptr(grad_lut), _ptr(grad_vol), _ptr(tmp), tmp_bytes, stream),
                   "mk_dvr_backward")
            return grad_vol, (grad_lut if ctx.needs_input_grad[1] else None), None

    return VolumeRender


_VR = None


def render(volume, lut, views):
    """Differentiable render of `views` (list of DVRParams): (V, H, W, 3)."""
    global _VR
    if _VR is None:
        _VR = _torch_function()
    return _VR.apply(volume, lut, list(views))
