"""The calls that a program built on this library makes, as timed cases.

Each case is one pass through a public entry point (capi.Volume, dvr.render,
server.Server) on a seeded CT-like phantom: air at -1000 HU, an ellipsoid body
at 40 HU with noise, dense spheres and vessels, labels on them where the case
has a mask -- the statistics of monkeygl_b200.phantom, generated on the GPU
because a 512x512x1559 volume takes too long on the host.  Camera angles,
planes, transfer functions and windows follow monkeygl_b200.workloads.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from monkeygl_b200 import capi, dvr, server, workloads
from monkeygl_b200.camera import Camera
from monkeygl_b200.phantom import Phantom, catmull_rom, make_tf_control_points, make_tf_lut

WW, WL = 1700.0, 650.0      # the CT window of every workload: [-200, 1500] HU

# ----------------------------------------------------------------------
# the cases

CARDIAC = dict(x=512, y=512, z=361, sx=0.351, sy=0.351, sz=0.3)
BODY = dict(x=512, y=512, z=1559, sx=0.7422, sy=0.7422, sz=1.0)


def listed():
    return [
        # a preview of a small volume while the user turns it: the smallest
        # call, where launches and the longest ray count
        dict(name="vr_small", kind="vr", x=128, y=128, z=96, sx=0.35, sy=0.35, sz=0.3, width=512, height=512,
             angle=45.0, tilt=0.0, zoom=1.0, labels=False, dense=False, rgba=False),
        # a rotating cardiac study at full screen size, left on the device
        dict(name="vr_cardiac", kind="vr", **CARDIAC, width=1024, height=1024, angle=30.0, tilt=0.0, zoom=1.0,
             labels=False, dense=False, rgba=False),
        # a whole-body CT with four segmented objects, opacity caps on all labels
        dict(name="vr_body", kind="vr", **BODY, width=1024, height=1024, angle=20.0, tilt=0.0, zoom=1.0,
             labels=True, dense=False, rgba=False),
        # the same study with soft tissue visible, where every ray composites
        # all through the body; zoomed and tilted, RGBA for a compositor
        dict(name="vr_dense", kind="vr", **BODY, width=1024, height=1024, angle=70.0, tilt=20.0, zoom=1.3,
             labels=True, dense=True, rgba=True),
        # the user drags the window/level: every frame follows a change of the
        # label parameters and goes back to the host; odd sizes
        dict(name="vr_drag", kind="drag", x=401, y=377, z=283, sx=0.7, sy=0.7, sz=0.8, width=637, height=479,
             angle=110.0, tilt=-15.0, zoom=1.1, labels=True, dense=False, rgba=False),
        # maximum intensity projection of the cardiac study
        dict(name="mip_cardiac", kind="mip", **CARDIAC, width=1024, height=1024, angle=60.0, tilt=0.0, zoom=1.0,
             labels=False, windows=False),
        # a viewer's three orthogonal planes after a cross-hair move, on the host
        dict(name="mpr_trio", kind="planes", **CARDIAC, width=512, height=512, half=0, mode=0, nearest=False,
             oblique=False),
        # a thick oblique slab (mean of 21 samples)
        dict(name="mpr_slab", kind="planes", x=512, y=512, z=600, sx=0.7, sy=0.7, sz=0.8, width=512, height=512,
             half=10, mode=0, nearest=False, oblique=True),
        # straightened curved reformat along a vessel of the whole-body study
        dict(name="cpr_body", kind="cpr", **BODY, width=512, height=1024, stretched=False),
        # a burst of mixed requests from several clients over resident volumes
        dict(name="serve_mix", kind="serve", requests=16, x=512, y=512, z=361, small=256),
        # one optimisation step of the differentiable renderer: 8 views, loss,
        # gradients of the volume and of the transfer function
        dict(name="dvr_train", kind="dvr", x=256, y=256, z=256, width=256, height=256, views=8, lut=256, step=0.5,
             angle=10.0, grads=True),
        # one view of an odd-sized volume without gradients
        dict(name="dvr_view", kind="dvr", x=211, y=190, z=157, width=321, height=243, views=1, lut=128, step=0.5,
             angle=35.0, grads=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above (sizes uniform in their logarithm)."""
    kind = rng.choice(["vr", "vr", "vr", "drag", "mip", "mip", "surface", "planes", "planes", "cpr", "serve", "dvr",
                       "dvr"])
    if kind == "dvr":
        x, y, z = (_log(rng, 40, 256) for _ in range(3))
        return dict(kind=kind, x=x, y=y, z=z, width=_log(rng, 32, 256), height=_log(rng, 32, 256),
                    views=_log(rng, 1, 8), lut=rng.choice([16, 64, 128, 256, 500]),
                    step=round(rng.uniform(0.5, 1.0), 2), angle=round(rng.uniform(0, 360), 1),
                    grads=rng.random() < 0.6)
    if kind == "serve":
        return dict(kind=kind, requests=rng.randint(2, 16), x=_log(rng, 96, 512), y=_log(rng, 96, 512),
                    z=_log(rng, 64, 361), small=_log(rng, 64, 256))
    size = dict(x=_log(rng, 64, 512), y=_log(rng, 64, 512), z=_log(rng, 48, 1559),
                sx=round(rng.uniform(0.3, 0.8), 3), sz=round(rng.uniform(0.3, 1.0), 2))
    size["sy"] = size["sx"]
    if kind == "cpr":
        return dict(kind=kind, **size, width=_log(rng, 64, 512), height=_log(rng, 128, 1024),
                    stretched=rng.random() < 0.5)
    size.update(width=_log(rng, 128, 1024), height=_log(rng, 128, 1024))
    if kind == "planes":
        return dict(kind=kind, **size, half=rng.choice([0, 0, 0, 2, 5, 10]), mode=rng.randrange(3),
                    nearest=rng.random() < 0.3, oblique=rng.random() < 0.6)
    view = dict(angle=round(rng.uniform(0, 360), 1), tilt=round(rng.uniform(-40, 40), 1),
                zoom=round(rng.uniform(0.8, 1.5), 2), labels=rng.random() < 0.5)
    if kind == "mip":
        return dict(kind=kind, **size, **view, windows=rng.random() < 0.3)
    if kind == "surface":
        return dict(kind=kind, **size, **view)
    return dict(kind=kind, **size, **view, dense=rng.random() < 0.25, rgba=rng.random() < 0.3)


# ----------------------------------------------------------------------
# inputs

def _phantom(dims, spacing, seed, labels=False):
    """Volume (and labels) as host arrays, and the vessels' control points."""
    X, Y, Z = dims
    dev = "cuda"
    rng = np.random.Generator(np.random.PCG64(seed))
    gen = torch.Generator(dev).manual_seed(seed)
    centre = np.array([X - 1, Y - 1, Z - 1]) / 2.0
    axes = np.array([0.45 * X, 0.40 * Y, 0.45 * Z])
    xs = ((torch.arange(X, device=dev) - centre[0]) / axes[0]) ** 2
    ys = ((torch.arange(Y, device=dev) - centre[1]) / axes[1]) ** 2
    zs = ((torch.arange(Z, device=dev) - centre[2]) / axes[2]) ** 2
    vol = torch.empty((Z, Y, X), dtype=torch.int16, device=dev)
    for z0 in range(0, Z, 128):
        z1 = min(Z, z0 + 128)
        noise = torch.randn((z1 - z0, Y, X), generator=gen, device=dev)
        inside = xs[None, None, :] + ys[None, :, None] + zs[z0:z1, None, None] <= 1.0
        vol[z0:z1] = torch.where(inside, torch.round(40.0 + 20.0 * noise), -1000.0).to(torch.int16)
    lab = torch.zeros((Z, Y, X), dtype=torch.uint8, device=dev) if labels else None

    def point(limit):
        while True:
            p = rng.uniform(0, 1, 3) * np.array([X - 1, Y - 1, Z - 1])
            if (((p - centre) / axes) ** 2).sum() <= limit:
                return p

    def paint(points, r, value, label):
        k = int(math.ceil(r)) + 1
        o = torch.arange(-k, k + 1, device=dev)
        off = torch.stack(torch.meshgrid(o, o, o, indexing="ij"), -1).reshape(1, -1, 3)
        p = torch.tensor(np.asarray(points).reshape(-1, 1, 3), device=dev)
        v = torch.floor(p).long() + off
        ok = ((v - p) ** 2).sum(-1) <= r * r
        for a, d in enumerate((X, Y, Z)):
            ok &= (v[..., a] >= 0) & (v[..., a] < d)
        v = v[ok]
        at = (v[:, 2], v[:, 1], v[:, 0])
        vol[at] = value
        if lab is not None:
            lab[at] = label

    for i in range(6):
        r, hu = rng.uniform(4.0, 10.0), rng.uniform(300.0, 1500.0)
        paint(point(0.6), r, int(hu), 1 if i < 3 else 2)
    vessels = []
    for j in range(3):
        r, hu = rng.uniform(2.0, 3.0), rng.uniform(250.0, 400.0)
        pts = np.array([point(0.7) for _ in range(6)])
        pts = pts[np.argsort(pts[:, 2])]
        vessels.append(pts)
        curve = catmull_rom(pts, 32)
        seg = np.linalg.norm(np.diff(curve, axis=0), axis=1)
        s = np.concatenate([[0.0], np.cumsum(seg)])
        t = np.linspace(0.0, s[-1], max(2, int(s[-1] / 0.5)))
        paint(np.stack([np.interp(t, s, curve[:, k]) for k in range(3)], 1), r, int(hu), 3 if j == 0 else 4)
    return Phantom(volume=vol.cpu().numpy(), spacing=spacing, labels=lab.cpu().numpy() if labels else None,
                   vessels=vessels)


def _camera(case, turn):
    c = Camera()
    c.anterior()
    c.rotate(case["angle"] + turn, case["tilt"])
    c.zoom(case["zoom"])
    return c


def _dense_lut():
    """Soft tissue visible: alpha 0.03 at about 0 HU, 0.12 at 300 HU."""
    return make_tf_lut([(0.0, (0.8, 0.5, 0.4, 0.0)), (0.12, (0.85, 0.55, 0.45, 0.03)), (0.3, (0.9, 0.7, 0.6, 0.12)),
                        (1.0, (1.0, 0.95, 0.9, 0.9))])


def _prepare_rays(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed + 100))
    dims, spacing = (case["x"], case["y"], case["z"]), (case["sx"], case["sy"], case["sz"])
    ph = _phantom(dims, spacing, seed, case["labels"])
    vol = capi.Volume(ph.volume)
    n = 1
    if case["labels"]:
        vol.set_mask(ph.labels)
        n = 5
    params = np.zeros((capi.MAX_LABELS, 3), np.float32)
    params[:, 1] = 1.0
    for l in range(n):
        lut = make_tf_lut(make_tf_control_points(rng))
        vol.set_transfer_function(l, _dense_lut() if case.get("dense") else lut)
        alpha = 1.0 if n == 1 else 0.4 if l == 0 else rng.uniform(0.6, 1.0)
        ww = WW + 40.0 * l if case.get("windows") else WW
        params[l] = (alpha, ww, WL)
    vol.set_label_params(params)
    kind = {"vr": capi.RENDER_VR, "drag": capi.RENDER_VR, "mip": capi.RENDER_MIP, "surface": capi.RENDER_SURFACE}
    rgba = bool(case.get("rgba"))
    p = capi.vr_params(case["width"], case["height"], kind[case["kind"]], _camera(case, float(rng.uniform(-5, 5))),
                       dims, spacing, pixel_format=capi.PIXEL_RGBA8 if rgba else capi.PIXEL_RGB8)
    shape = (case["height"], case["width"], 4 if rgba else 3)
    if case["kind"] == "drag":
        return dict(kind="drag", vol=vol, p=p, params=params, out=np.empty(shape, np.uint8))
    return dict(kind="rays", vol=vol, p=p, out=torch.empty(shape, dtype=torch.uint8, device="cuda"))


def _prepare_planes(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed + 100))
    dims, spacing = (case["x"], case["y"], case["z"]), (case["sx"], case["sy"], case["sz"])
    ph = _phantom(dims, spacing, seed)
    ext, ps = np.array(dims) * np.array(spacing), min(spacing)
    W, H = case["width"], case["height"]
    if case["oblique"]:
        n = rng.standard_normal(3)
        n /= np.linalg.norm(n)
        h = np.cross(n, [1.0, 0, 0] if abs(n[0]) < 0.9 else [0, 1.0, 0])
        h /= np.linalg.norm(h)
        frames = [(h, np.cross(n, h))]
    else:
        frames = [([1.0, 0, 0], [0, 1.0, 0]), ([0, 1.0, 0], [0, 0, -1.0]), ([1.0, 0, 0], [0, 0, -1.0])]
    centre = ext / 2 + rng.uniform(-0.1, 0.1, 3) * ext
    planes = []
    for h, v in frames:
        h, v = np.array(h), np.array(v)
        lt = centre - h * (0.5 * W * ps) - v * (0.5 * H * ps)
        planes.append(capi.plane_params(W, H, case["mode"], int(case["nearest"]), spacing, h, v, np.cross(h, v), lt,
                                        ps, False, case["half"]))
    return dict(kind="planes", vol=capi.Volume(ph.volume), planes=planes,
                outs=[np.empty((H, W), np.int16) for _ in planes])


def _prepare_cpr(case, seed):
    dims, spacing = (case["x"], case["y"], case["z"]), (case["sx"], case["sy"], case["sz"])
    ph = _phantom(dims, spacing, seed)
    path = workloads.vessel_path(ph, n_points=200, rows=case["height"])
    build = workloads.cpr_stretched if case["stretched"] else workloads.cpr_straightened
    pts, dirs = build(path, case["width"])
    return dict(kind="cpr", vol=capi.Volume(ph.volume), width=case["width"], pts=np.ascontiguousarray(pts),
                dirs=np.ascontiguousarray(dirs), out=np.empty((case["height"], case["width"]), np.int16))


def _prepare_serve(case, seed):
    s = case["small"]
    shapes = [((s, s, s), (1.0, 1.0, 1.0), False), ((case["x"], case["y"], case["z"]), (0.351, 0.351, 0.3), False),
              ((s + 41, s + 19, s + 85), (0.7, 0.7, 0.8), True)]
    srv = server.Server(hbm_budget_bytes=6 << 30, max_bricks=1 << 18)
    ids = []
    for i, (dims, spacing, labels) in enumerate(shapes):
        ph = _phantom(dims, spacing, seed + i, labels)
        ids.append(srv.add_volume(ph.volume, ph.labels))
    reqs, outs = [], []
    for i in range(case["requests"]):       # of ten: six VR, one MIP, one surface, two planes
        size, mix = (256, 512, 768, 1024)[i % 4], (0, 0, 1) if i % 5 == 3 else (0, 1, 0) if i % 5 == 1 else (1, 0, 0)
        r = workloads.serving_trace([shapes[i % 3]], 1, 1000.0, seed=100 * seed + i, sizes=(size,), mix=mix)[0]
        r.volume = i % 3
        if r.kind == capi.REQUEST_MIP and i % 2:
            r.kind = capi.REQUEST_SURFACE
        reqs.append(r)
        outs.append(server._pinned_empty((size, size), np.int16)[0] if r.kind == capi.REQUEST_MPR else
                    server._pinned_empty((size, size, 3), np.uint8)[0])
    return dict(kind="serve", srv=srv, ids=ids, reqs=reqs, outs=outs)


def _dvr_inputs(case, seed):
    dims = (case["x"], case["y"], case["z"])
    rng = np.random.Generator(np.random.PCG64(seed + 100))
    ph = _phantom(dims, (1.0, 1.0, 1.0), seed)
    vol = torch.from_numpy(ph.volume).cuda().float().add_(1024.0).div_(4095.0).clamp_(0.0, 1.0)
    lut = torch.tensor(make_tf_lut(make_tf_control_points(rng), case["lut"]), device="cuda")
    views = []
    for i in range(case["views"]):
        c = Camera()
        c.anterior()
        c.rotate(case["angle"] + i * 360.0 / case["views"], 0.0)
        views.append(dvr.dvr_params(case["width"], case["height"], c, dims, (1, 1, 1), case["step"], 1e-4,
                                    case["lut"]))
    target = None
    if case["grads"]:
        gen = torch.Generator("cuda").manual_seed(seed)
        target = torch.rand((case["views"], case["height"], case["width"], 3), generator=gen, device="cuda")
    return vol, lut, views, target


def _prepare_dvr(case, seed):
    vol, lut, views, target = _dvr_inputs(case, seed)
    if case["grads"]:
        vol.requires_grad_()
        lut.requires_grad_()
    return dict(kind="dvr", vol=vol, lut=lut, views=views, target=target)


def prepare(case, seed):
    make = {"planes": _prepare_planes, "cpr": _prepare_cpr, "serve": _prepare_serve, "dvr": _prepare_dvr}
    return make.get(case["kind"], _prepare_rays)(case, seed)


# ----------------------------------------------------------------------
# one pass

def _stream():
    # 1 names CUDA's legacy default stream, torch's own unless one is set: the
    # image is then ordered with the torch work around it
    return torch.cuda.current_stream().cuda_stream or 1


def run(s):
    kind = s["kind"]
    if kind == "rays":
        s["vol"].render_vr_device(s["p"], s["out"].data_ptr(), _stream())
        return s["out"]
    if kind == "drag":
        s["vol"].set_label_params(s["params"])
        return s["vol"].render_vr(s["p"], out=s["out"])
    if kind == "planes":
        return [s["vol"].render_plane(p, out=o) for p, o in zip(s["planes"], s["outs"])]
    if kind == "cpr":
        return s["vol"].render_cpr(s["width"], s["pts"], s["dirs"], False, out=s["out"])
    if kind == "serve":
        tickets = [server.submit_request(s["srv"], s["ids"][r.volume], r, out=o) for r, o in zip(s["reqs"], s["outs"])]
        return [s["srv"].wait(t)[0] for t in tickets]
    images = dvr.render(s["vol"], s["lut"], s["views"])
    if s["target"] is None:
        return images
    loss = ((images - s["target"]) ** 2).mean()
    g_vol, g_lut = torch.autograd.grad(loss, (s["vol"], s["lut"]))
    return {"images": images.detach(), "grad_volume": g_vol, "grad_lut": g_lut}


def work(case):
    """Bytes: the volume (and labels) read once where the path looks at all of
    it, the voxels about the plane where it does not, and the outputs written
    once.  Flops: about 60 a sample of the path's own sampling."""
    kind = case["kind"]
    if kind == "serve":
        vox = 2 * case["small"] ** 3 + case["x"] * case["y"] * case["z"]
        return {"bytes": 2.0 * vox + case["requests"] * 3.0 * 512 * 512, "flops": 0.0}
    vox, pix = case["x"] * case["y"] * case["z"], case["width"] * case["height"]
    if kind == "dvr":
        samples = case["views"] * pix * 0.5 * case["z"] / case["step"]
        back = case["grads"]
        return {"bytes": 4.0 * vox * (2 if back else 1) + 12.0 * pix * case["views"] * (2 if back else 1),
                "flops": samples * (60 + (90 if back else 0))}
    if kind == "planes":
        n = 1 if case["oblique"] else 3
        taps = n * pix * (2 * case["half"] + 1)
        return {"bytes": min(2.0 * vox, 2.0 * 2 * taps) + 2.0 * n * pix, "flops": 40.0 * taps}
    if kind == "cpr":
        return {"bytes": 2.0 * 2 * pix + 2.0 * pix, "flops": 40.0 * pix}
    return {"bytes": vox * (3.0 if case["labels"] else 2.0) + pix * (4.0 if case.get("rgba") else 3.0), "flops": 0.0}


# ----------------------------------------------------------------------
# the differentiable renderer in 64 bits (the other cases give whole numbers)

def _view64(p, vol, lut):
    """The samples of every ray of one view: a function of the step number."""
    W, H, f32 = p.width, p.height, np.float32
    dev, f64 = vol.device, torch.float64
    dims = torch.tensor(list(p.dims), dtype=f64, device=dev)
    M = torch.tensor(list(p.transform), dtype=f64, device=dev).view(3, 3)
    mls = torch.tensor(list(p.max_len_spacing), dtype=f64, device=dev)
    ys, xs = torch.meshgrid(torch.arange(H, device=dev, dtype=f64), torch.arange(W, device=dev, dtype=f64),
                            indexing="ij")
    u, v = (xs - W / 2.0 - p.x_translate) / H, (ys - H / 2.0 - p.y_translate) / H
    uvw = torch.stack([u, torch.full_like(u, -float(f32(0.866)) * p.scale), v], -1).view(-1, 3)
    base, step = (uvw @ M.T) * mls + 0.5, M[:, 1] * p.scale * mls
    lo, hi = torch.zeros(W * H, dtype=f64, device=dev), torch.full((W * H,), float(f32(1.732)), dtype=f64, device=dev)
    hit = torch.ones(W * H, dtype=torch.bool, device=dev)
    for k in range(3):
        if abs(step[k].item()) < 1e-12:
            hit &= (base[:, k] >= 0) & (base[:, k] <= 1)
            continue
        a, b = (0.0 - base[:, k]) / step[k], (1.0 - base[:, k]) / step[k]
        lo, hi = torch.maximum(lo, torch.minimum(a, b)), torch.minimum(hi, torch.maximum(a, b))
    first = torch.ceil(lo / p.step) * p.step
    count = torch.where(hit & (lo < hi), (torch.floor((hi - first) / p.step) + 1).clamp(min=0), 0.0).long()
    n = lut.shape[0]

    def sample(i):
        c = (base + (first + i * p.step)[:, None] * step) * dims - 0.5
        f = torch.floor(c)
        w, f = c - f, f.long()
        at, wt, s = [], [], 0.0
        for corner in range(8):
            q, t = [], 1.0
            for k in range(3):
                bit = corner >> k & 1
                q.append((f[:, k] + bit).clamp(0, p.dims[k] - 1))
                t = t * (w[:, k] if bit else 1.0 - w[:, k])
            at.append((q[2] * p.dims[1] + q[1]) * p.dims[0] + q[0])
            wt.append(t)
            s = s + t * vol.view(-1)[at[-1]]
        x = s * n - 0.5
        inside = (x >= 0) & (x < n - 1)
        x = x.clamp(0, n - 1)
        k0 = x.long()
        k1 = (k0 + 1).clamp(max=n - 1)
        return at, wt, inside, k0, k1, (x - k0)[:, None]

    return sample, count


def exact(case, seed):
    if case["kind"] != "dvr":
        return None
    vol, lut, views, target = _dvr_inputs(case, seed)
    vol, lut, n = vol.double(), lut.double(), case["lut"]
    g_vol, g_lut = torch.zeros_like(vol).view(-1), torch.zeros_like(lut)
    images = torch.zeros((case["views"], case["height"], case["width"], 3), dtype=torch.float64, device="cuda")
    for j, p in enumerate(views):
        sample, count = _view64(p, vol, lut)
        colour = images[j].view(-1, 3)
        T, live, Ts = torch.ones(len(count), dtype=torch.float64, device="cuda"), count > 0, []
        for i in range(int(count.max())):
            _, _, _, k0, k1, w = sample(i)
            c = lut[k0] + w * (lut[k1] - lut[k0])
            a = torch.where(live, c[:, 3], 0.0)
            Ts.append(torch.where(live, T, 0.0))
            colour += (T * a)[:, None] * c[:, :3]
            T = T * (1.0 - a)
            live = live & (i + 1 < count) & (T >= p.t_min)
        if target is None:
            continue
        g = 2.0 * (colour - target[j].double().view(-1, 3)) / target.numel()
        U = torch.zeros_like(colour)
        for i in reversed(range(len(Ts))):
            at, wt, inside, k0, k1, w = sample(i)
            d = lut[k1] - lut[k0]
            c = lut[k0] + w * d
            T, a = Ts[i], torch.where(Ts[i] > 0, c[:, 3], 0.0)
            gc = torch.cat([(T * a)[:, None] * g, (T * (g * (c[:, :3] - U)).sum(1))[:, None]], 1)
            U = a[:, None] * c[:, :3] + (1.0 - a)[:, None] * U
            g_lut.index_add_(0, k0, (1.0 - w) * gc)
            g_lut.index_add_(0, k1, w * gc)
            gs = torch.where(inside, n * (gc * d).sum(1), 0.0)
            for q, t in zip(at, wt):
                g_vol.index_add_(0, q, t * gs)
    if target is None:
        return images
    return {"images": images, "grad_volume": g_vol.view_as(vol), "grad_lut": g_lut}
