"""The work that users of this framework have it do, as measurable cases.

A registration of a CT volume to X-ray images asks for: DRRs of candidate poses, the similarity of each to
the fixed image, populations of such poses (one job or several), and, once per patient and view, the set-up
of the volume and of the fixed images.  Every case goes through the package's public entry points.

Inputs are made on the GPU from the seed alone: an ellipsoidal body with bones and noise (the phantom of the
benchmark), poses about a nominal view, fixed images drawn with torch.  `exact` restates the results in
64 bits with torch only.
"""
import math
import random

import numpy as np
import torch
import torch.nn.functional as F

import xreg_gb300 as xr

SDD, SOD, PANEL = 1020.0, 700.0, 298.0  # mm: source to detector, source to volume centre, detector edge
VOXEL = {"f32": 0, "f16": 1, "bf16": 2}
METRICS = {"ncc": xr.ImgSimMetric2DNCCCUDA, "grad_ncc": xr.ImgSimMetric2DGradNCCCUDA,
           "patch_ncc": xr.ImgSimMetric2DPatchNCCCUDA, "patch_grad_ncc": xr.ImgSimMetric2DPatchGradNCCCUDA}
MU_W, MU_A = 0.02683, 0.02485e-4


# ------------------------------------------------------------------ the cases
def _objective(name, size, sxy, sz, det, views, pop, dtype, metric, air="clean", rot=10.0, trans=20.0, mask=False):
    return {"name": name, "kind": "objective", "nx": size[0], "ny": size[1], "nz": size[2], "sxy": sxy, "sz": sz,
            "rows": det[0], "cols": det[1], "views": views, "pop": pop, "dtype": dtype, "metric": metric, "air": air,
            "step": 0.5, "rot": rot, "trans": trans, "mask": mask}


def listed():
    return [
        # one DRR and its NCC through the ray caster's and the metric's own calls, a value read per pose: code
        # written against the operators (the plain method), where launches and latency count
        {"name": "plain-ncc", "kind": "operators", "nx": 128, "ny": 128, "nz": 128, "sxy": 1.5, "sz": 1.5,
         "rows": 256, "cols": 256, "views": 1, "pop": 1, "dtype": "f32", "metric": "ncc", "air": "clean",
         "step": 0.5, "rot": 5.0, "trans": 10.0, "mask": False},
        # one candidate of a two-view fine level: the BOBYQA stage asks for one point at a time
        _objective("fine-point", (256, 256, 200), 300.0 / 256, 300.0 / 256, (384, 384), 2, 1, "f16", "grad_ncc",
                   rot=1.0, trans=2.0),
        # a CMA-ES generation of a coarse level (detector downsampled 8x), three views
        _objective("coarse-population", (320, 320, 256), 300.0 / 320, 300.0 / 320, (192, 192), 3, 57, "f16", "grad_ncc"),
        # the benchmark's population: 256^3, detector downsampled 4x, lambda 100, float32 voxels
        _objective("population", (256, 256, 256), 1.0, 1.0, (384, 384), 1, 100, "f32", "grad_ncc"),
        # CT as scanners give it: noisy air keeps about half of its voxels positive, so little can be skipped;
        # odd sizes after cropping, a masked field of view
        _objective("noisy-air-population", (251, 243, 237), 1.0, 1.0, (383, 381), 1, 40, "f32", "grad_ncc",
                   air="noisy", mask=True),
        # bfloat16 voxels, the plain NCC, two views
        _objective("bf16-population", (256, 256, 200), 300.0 / 256, 300.0 / 256, (300, 260), 2, 24, "bf16", "ncc"),
        # the finest level: a full-size CT in half precision, 768^2 views, patch grad-NCC 11x11
        _objective("patch-population", (512, 512, 400), 0.8, 1.0, (768, 768), 1, 20, "f16", "patch_grad_ncc", rot=5.0,
                   trans=10.0),
        # four registrations of uneven size evaluated in one call: a step of the serving loop
        {"name": "uneven-jobs", "kind": "jobs", "jobs": 4, "mix": 4, "dtype": "f16", "step": 0.5},
        # a new patient: HU to attenuation, the volume's layouts, and a DRR of each view
        {"name": "admit-volume", "kind": "admit", "nx": 512, "ny": 512, "nz": 300, "sxy": 300.0 / 512,
         "sz": 300.0 / 512, "rows": 384, "cols": 384, "views": 2, "pop": 1, "dtype": "f16", "air": "clean",
         "step": 0.5, "rot": 5.0, "trans": 10.0},
        # a new X-ray image: crop, log remap, and the images of two registration levels, from and to host arrays
        {"name": "prepare-xray", "kind": "xray", "rows": 1536, "cols": 1536, "f1": 0.25, "f2": 0.125},
        # a masked, patch-wise comparison of given images (no ray casting)
        {"name": "masked-patches", "kind": "images", "metric": "patch_ncc", "rows": 384, "cols": 384, "n": 24,
         "radius": 5, "stride": 2, "mask": True},
        # full-resolution DRRs to the host: what synthetic fixed images and visual checks are made of
        {"name": "full-resolution-drr", "kind": "render", "nx": 256, "ny": 256, "nz": 256, "sxy": 1.0, "sz": 1.0,
         "rows": 1536, "cols": 1536, "views": 1, "pop": 1, "dtype": "f32", "line": "sum", "air": "clean", "step": 0.5,
         "rot": 5.0, "trans": 10.0},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["operators", "objective", "objective", "objective", "objective", "jobs", "admit", "xray",
                       "images", "render"])
    if kind == "jobs":
        return {"kind": kind, "jobs": rng.randint(2, 4), "mix": rng.randint(10, 10 ** 6),
                "dtype": rng.choice(["f16", "f16", "f32", "bf16"]), "step": 0.5}
    if kind == "xray":
        return {"kind": kind, "rows": int(_log(rng, 480, 1536)), "cols": int(_log(rng, 480, 1536)),
                "f1": rng.choice([0.5, 0.25, 0.3]), "f2": rng.choice([0.125, 0.2])}
    if kind == "images":
        metric = rng.choice(list(METRICS))
        return {"kind": kind, "metric": metric, "rows": int(_log(rng, 96, 500)), "cols": int(_log(rng, 96, 500)),
                "n": int(_log(rng, 1, 40)), "radius": rng.choice([3, 5, 5, 7]), "stride": rng.choice([1, 2, 3]),
                "mask": rng.random() < 0.5}
    c = {"kind": kind}
    for a in ("nx", "ny", "nz"):
        c[a] = int(_log(rng, 120, 420))
    c["sxy"] = 300.0 / c["nx"] if rng.random() < 0.5 else rng.choice([0.8, 1.0, 1.2])
    c["sz"] = c["sxy"] if rng.random() < 0.6 else rng.choice([0.8, 1.0, 1.5])
    big = 1400 if kind == "render" else 640
    c["rows"] = int(_log(rng, 128, big))
    c["cols"] = max(128, min(big, int(c["rows"] * rng.uniform(0.8, 1.25))))
    c["views"] = rng.choice([1, 1, 2, 3])
    c["dtype"] = rng.choice(["f32", "f16", "f16", "bf16"])
    c["air"] = rng.choice(["clean", "clean", "noisy"])
    c["step"] = rng.choice([0.5, 0.5, 1.0])
    c["rot"], c["trans"] = rng.choice([(10.0, 20.0), (5.0, 10.0), (1.0, 2.0)])
    c["pop"] = 1
    if kind in ("operators", "objective"):
        c["metric"] = rng.choice(["ncc", "grad_ncc", "grad_ncc", "patch_ncc", "patch_grad_ncc"])
        c["mask"] = rng.random() < 0.25
    if kind == "operators":
        c["views"] = 1
    if kind == "render":
        c["line"] = rng.choice(["sum", "sum", "max"])
    if kind == "objective":
        top = _samples(listed()[3], 1) * 100 / _samples(c, 1)  # no more work than the benchmark's population
        if c["metric"].startswith("patch"):
            top = min(top, 20 * 768 * 768 / (c["rows"] * c["cols"] * c["views"]))
        c["pop"] = max(1, int(_log(rng, 1, max(1.5, min(100, top)))))
    return c


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _hu(size, sp, seed, air="clean"):
    """HU volume [nz, ny, nx]: soft tissue with noise in an ellipsoid, 3 to 5 bones, air of -1000 HU (noisy: +- 10 HU)."""
    r = random.Random(int(seed))
    ext = [n * s for n, s in zip(size, sp)]
    c = [e * (0.5 + r.uniform(-0.02, 0.02)) for e in ext]
    a = [ext[0] * r.uniform(0.40, 0.46), ext[1] * r.uniform(0.30, 0.38), ext[2] * r.uniform(0.42, 0.47)]
    ax = [torch.arange(n, device="cuda", dtype=torch.float32) * s for n, s in zip(size, sp)]
    X, Y, Z = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]

    def inside(c, a):
        return ((X - c[0]) / a[0]) ** 2 + ((Y - c[1]) / a[1]) ** 2 + ((Z - c[2]) / a[2]) ** 2 <= 1.0

    body = inside(c, a)
    hu = torch.where(body, r.uniform(0.0, 60.0), -1000.0).float()
    for _ in range(r.randint(3, 5)):
        bc = [u + r.uniform(-0.55, 0.55) * v for u, v in zip(c, a)]
        ba = [e * r.uniform(0.04, 0.14) for e in ext]
        hu = torch.where(inside(bc, ba) & body, r.uniform(300.0, 1500.0), hu)
    noise = torch.randn(hu.shape, device="cuda", generator=_gen(seed + 1)) * 10.0
    hu += noise if air == "noisy" else noise * body
    return hu.contiguous()


def _mu64(hu):
    """HUToLinAtt in double."""
    scale = (MU_W - MU_A) * 1.0e-3
    return (hu.double() * scale + MU_W - (-1000.0 * scale + MU_W)).clamp_(min=0.0)


def _rigid(R, t):
    T = np.eye(4)
    T[:3, :3], T[:3, 3] = R, t
    return T


def _euler(x, y, z):
    cx, sx, cy, sy, cz, sz = math.cos(x), math.sin(x), math.cos(y), math.sin(y), math.cos(z), math.sin(z)
    return np.array([[cz, -sz, 0], [sz, cz, 0], [0, 0, 1]]) @ np.array([[cy, 0, sy], [0, 1, 0], [-sy, 0, cy]]) @ \
        np.array([[1, 0, 0], [0, cx, -sx], [0, sx, cx]])


def _poses(size, sp, n, rot, trans, seed):
    """Camera -> physical poses about the volume centre, rotations N(0, rot deg), translations N(0, trans mm)."""
    r = np.random.default_rng(int(seed) + 2)
    C = _rigid(np.eye(3), [k * s / 2.0 for k, s in zip(size, sp)])
    view = np.array([[1.0, 0, 0], [0, 0, 1.0], [0, -1.0, 0]])
    nominal = C @ _rigid(view, view @ np.array([0.0, 0.0, SOD]))
    out = np.empty((n, 4, 4))
    for k in range(n):
        D = _rigid(_euler(*np.radians(r.normal(0.0, rot, 3))), r.normal(0.0, trans, 3))
        out[k] = C @ D @ np.linalg.inv(C) @ nominal
    return out


def _extrins(view):
    """World -> camera of view k: 25 degrees more about the volume centre for each."""
    a = math.radians(25.0 * view)
    R = np.array([[math.cos(a), 0, math.sin(a)], [0, 1, 0], [-math.sin(a), 0, math.cos(a)]])
    c = np.array([0.0, 0.0, -SOD])
    return _rigid(R, c - R @ c)


def _cams(rows, cols, views):
    px = PANEL / max(rows, cols)
    cams = []
    for v in range(views):
        cam = xr.CameraModel.naive(SDD, rows, cols, px, px)
        if v:
            cam.set_extrins(_extrins(v))
        cams.append(cam)
    return cams


def _rays(size, sp, rows, cols, view, pose, step):
    """Start points, steps (index space, x y z) and sample counts of the step rule, [rows * cols], in double."""
    px = PANEL / max(rows, cols)
    Ei = np.linalg.inv(_extrins(view)) if view else np.eye(4)
    M = np.diag([1.0 / s for s in sp] + [1.0]) @ pose
    t = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
    r, c = torch.meshgrid(torch.arange(rows, device="cuda", dtype=torch.float64),
                          torch.arange(cols, device="cuda", dtype=torch.float64), indexing="ij")
    det = torch.stack([(c - (cols - 1) / 2) * px, (r - (rows - 1) / 2) * px, torch.full_like(r, -SDD)], -1).reshape(-1, 3)
    det = det @ t(Ei[:3, :3]).T + t(Ei[:3, 3])
    pin = t(Ei[:3, 3])
    a = M[:3, :3] @ Ei[:3, 3] + M[:3, 3]
    d = det @ t(M[:3, :3]).T + t(M[:3, 3]) - t(a)
    hi = t([n - 1.0 for n in size])
    inv = 1.0 / d
    ta, tb = (0.0 - t(a)) * inv, (hi - t(a)) * inv
    t0 = torch.minimum(ta, tb).amax(-1).clamp(min=0.0)
    t1 = torch.maximum(ta, tb).amin(-1).clamp(max=1.0)
    hit = t1 - t0 > 2.0e-3
    t0, t1 = t0 + 1.0e-3, t1 - 1.0e-3
    u = det - pin
    w = (u / u.norm(dim=-1, keepdim=True) * step) @ t(M[:3, :3]).T
    slen, dlen = w.norm(dim=-1), d.norm(dim=-1)
    n = torch.where(hit, ((t1 - t0) * dlen / slen).floor() + 1, 0.0)
    return t(a) + t0[:, None] * d, d * (slen / dlen)[:, None], n


def _drr(vol, size, sp, rows, cols, view, pose, step, line="sum", most=40_000_000):
    """One DRR of vol [nz, ny, nx] in vol's precision, by the step rule."""
    p0, st, n = _rays(size, sp, rows, cols, view, pose, step)
    p0, st = p0.to(vol.dtype), st.to(vol.dtype)
    out = torch.zeros(rows * cols, dtype=vol.dtype, device="cuda")
    top = int(n.max())
    if top <= 0:
        return out.view(rows, cols)
    scale = torch.tensor([2.0 / (k - 1) for k in size], dtype=vol.dtype, device="cuda")
    k = torch.arange(top, device="cuda", dtype=vol.dtype)
    rows_at_once = max(1, most // top)
    for b in range(0, rows * cols, rows_at_once):
        e = min(rows * cols, b + rows_at_once)
        g = (p0[b:e, None, :] + k[None, :, None] * st[b:e, None, :]) * scale - 1.0
        s = F.grid_sample(vol[None, None], g[None, None], mode="bilinear", padding_mode="border", align_corners=True)[0, 0, 0]
        s = torch.where(k[None] < n[b:e, None], s, 0.0)
        out[b:e] = (s.amax(-1) if line == "max" else s.sum(-1)) * step
    return out.view(rows, cols)


def _noisy(img, seed):
    return img + 0.01 * (img.max() - img.min()) * torch.randn(img.shape, device="cuda", generator=_gen(seed), dtype=img.dtype)


def _fixed(hu, size, sp, c, seed):
    """Fixed image of each view: float32 DRRs (1 mm step) at a pose near the nominal one, with 1 % noise."""
    vol = _mu64(hu).float()
    pose = _poses(size, sp, 1, 3.0, 5.0, seed + 50)[0]
    return [_noisy(_drr(vol, size, sp, c["rows"], c["cols"], v, pose, 1.0), seed + 60 + v).cpu().numpy()
            for v in range(c["views"])]


def _mask(rows, cols, seed):
    """A round field of view with a rectangle (an implant, a label) left out."""
    y, x = np.mgrid[0:rows, 0:cols]
    m = ((y - rows / 2) / (0.48 * rows)) ** 2 + ((x - cols / 2) / (0.48 * cols)) ** 2 <= 1.0
    r = random.Random(seed + 3)
    a, b = int(r.uniform(0.2, 0.6) * rows), int(r.uniform(0.2, 0.6) * cols)
    m[a:a + rows // 8, b:b + cols // 6] = False
    return m.astype(np.uint8)


class _Device:
    """A device pointer as torch sees it; owner, which holds the memory, lives as long as the tensor."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": tuple(shape), "typestr": "<f4", "version": 2}


def _images_of(rc, n, c):
    """The caster's projection buffer as a tensor (no copy)."""
    return torch.as_tensor(_Device(rc.device_pixel_buf(), (n, c["rows"], c["cols"]), rc), device="cuda")


def _geometry(c):
    return (c["nx"], c["ny"], c["nz"]), (c["sxy"], c["sxy"], c["sz"])


def _volume(size, sp):
    """The volume's geometry; its voxels are on the device (the host array is never touched)."""
    return xr.Volume(np.empty(size[::-1], np.float32), spacing=sp)


def _caster(c, hu):
    size, sp = _geometry(c)
    rc = xr.RayCasterLineIntCUDA()
    mu = _mu64(hu).float()
    torch.cuda.synchronize()
    rc.set_volumes_device([_volume(size, sp)], [mu.data_ptr()], VOXEL[c["dtype"]])
    rc.set_camera_models(_cams(c["rows"], c["cols"], c["views"]))
    rc.set_ray_step_size(c["step"])
    return rc


def _metrics(c, hu, seed):
    size, sp = _geometry(c)
    ms = []
    for f in _fixed(hu, size, sp, c, seed):
        m = METRICS[c["metric"]]()
        m.set_fixed_image(f)
        if c["mask"]:
            m.set_mask(_mask(c["rows"], c["cols"], seed))
        ms.append(m)
    return ms


def _job_cases(c):
    """The registrations of an uneven set: volumes from 192^3 to 448 x 448 x 300, 1 to 3 views, 4x or 8x, lambda 20 to 100."""
    r = random.Random(c["mix"])
    out = []
    for _ in range(c["jobs"]):
        size = r.choice([(192, 192, 192), (256, 256, 200), (256, 256, 256), (320, 320, 256), (384, 384, 280), (448, 448, 300)])
        views, det = r.randint(1, 3), r.choice([384, 192])
        top = 100 if det == 192 else 60 // views
        j = _objective("", size, 300.0 / size[0], 300.0 / size[0], (det, det), views, r.randint(20, max(20, top)), c["dtype"],
                       "grad_ncc")
        j["step"] = c["step"]
        out.append(j)
    return out


def _objective_state(c, seed):
    size, sp = _geometry(c)
    hu = _hu(size, sp, seed, c["air"])
    rc = _caster(c, hu)
    ms = _metrics(c, hu, seed)
    obj = xr.PopulationObjective(rc, ms, c["pop"])
    return {"rc": rc, "obj": obj, "poses": _poses(size, sp, c["pop"], c["rot"], c["trans"], seed),
            "drr": _images_of(rc, c["views"] * c["pop"], c)}


def _raw_xray(c, seed):
    """A raw detector image: exp(-line integrals) with noise, 16-bit counts."""
    small = _drr(_mu64(_hu((128, 128, 128), (2.0, 2.0, 2.0), seed)).float(), (128, 128, 128), (2.0, 2.0, 2.0), 192, 192, 0,
                 _poses((128, 128, 128), (2.0, 2.0, 2.0), 1, 3.0, 5.0, seed)[0], 1.0)
    img = F.interpolate(small[None, None], (c["rows"], c["cols"]), mode="bilinear", align_corners=False)[0, 0]
    img = 40000.0 * torch.exp(-img) * (1.0 + 0.01 * torch.randn(img.shape, device="cuda", generator=_gen(seed + 5)))
    return img.round_().clamp_(0.0, 65535.0).cpu().numpy()


def _given_images(c, seed):
    """n moving DRRs of a small volume about a pose, and the fixed image at it."""
    size, sp = (96, 96, 96), (2.5, 2.5, 2.5)
    vol = _mu64(_hu(size, sp, seed)).float()
    imgs = torch.stack([_drr(vol, size, sp, c["rows"], c["cols"], 0, p, 2.0) for p in _poses(size, sp, c["n"] + 1, 3.0, 5.0, seed)])
    return _noisy(imgs[0], seed + 4).contiguous(), imgs[1:].contiguous()


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "objective":
        return dict(_objective_state(c, seed), kind=kind)
    if kind == "jobs":
        jobs = [_objective_state(j, seed + 1000 * k) for k, j in enumerate(_job_cases(c))]
        return {"kind": kind, "jobs": jobs, "set": xr.JobSet()}
    if kind == "operators":
        size, sp = _geometry(c)
        hu = _hu(size, sp, seed, c["air"])
        rc = _caster(c, hu)
        rc.set_num_projs(1)
        rc.allocate_resources()
        m = _metrics(c, hu, seed)[0]
        m.set_num_moving_images(1)
        m.set_mov_imgs_buf_from_ray_caster(rc, 0)
        m.allocate_resources()
        return {"kind": kind, "rc": rc, "m": m, "poses": _poses(size, sp, 1, c["rot"], c["trans"], seed), "drr": _images_of(rc, 1, c)}
    if kind == "render":
        size, sp = _geometry(c)
        rc = _caster(c, _hu(size, sp, seed, c["air"]))
        rc.set_kernel_id(1 if c["line"] == "max" else 0)
        rc.set_num_projs(c["views"])
        rc.allocate_resources()
        return {"kind": kind, "rc": rc, "poses": _poses(size, sp, 1, c["rot"], c["trans"], seed)}
    if kind == "admit":
        size, sp = _geometry(c)
        hu = _hu(size, sp, seed, c["air"])
        stream = torch.cuda.Stream()
        rc = xr.RayCasterLineIntCUDA()
        rc.set_stream(stream.cuda_stream)
        rc.set_camera_models(_cams(c["rows"], c["cols"], c["views"]))
        rc.set_ray_step_size(c["step"])
        rc.set_num_projs(c["views"])
        rc.allocate_resources()
        torch.cuda.synchronize()
        return {"kind": kind, "rc": rc, "stream": stream, "hu": hu, "mu": torch.empty_like(hu), "vol": _volume(size, sp),
                "dtype": VOXEL[c["dtype"]], "poses": _poses(size, sp, 1, c["rot"], c["trans"], seed),
                "drr": _images_of(rc, c["views"], c)}
    if kind == "xray":
        px = PANEL / max(c["rows"], c["cols"])
        return {"kind": kind, "raw": _raw_xray(c, seed), "cam": xr.CameraModel.naive(SDD, c["rows"], c["cols"], px, px),
                "f": (c["f1"], c["f2"])}
    fixed, mov = _given_images(c, seed)
    torch.cuda.synchronize()
    m = METRICS[c["metric"]]()
    m.set_fixed_image(fixed.cpu().numpy())
    if c["mask"]:
        m.set_mask(_mask(c["rows"], c["cols"], seed))
    if c["metric"].startswith("patch"):
        m.set_patch_radius(c["radius"])
        m.set_patch_stride(c["stride"])
    m.set_num_moving_images(c["n"])
    m.set_mov_imgs_device_buf(mov.data_ptr())
    m.allocate_resources()
    return {"kind": kind, "m": m, "mov": mov}


def run(s):
    kind = s["kind"]
    if kind == "objective":
        return {"sims": s["obj"].eval(s["poses"]), "drr": s["drr"]}
    if kind == "jobs":
        sims = s["set"].eval([j["obj"] for j in s["jobs"]], [j["poses"] for j in s["jobs"]])
        return {"sims": sims, "drr": [j["drr"] for j in s["jobs"]]}
    if kind == "operators":
        s["rc"].distribute_xforms_among_cam_models(s["poses"])
        s["rc"].compute()
        s["m"].compute()
        return {"sims": s["m"].sim_vals(), "drr": s["drr"]}
    if kind == "render":
        s["rc"].distribute_xforms_among_cam_models(s["poses"])
        s["rc"].compute()
        return s["rc"].projs()
    if kind == "admit":
        rc = s["rc"]
        xr.hu_to_lin_att_device(s["hu"].data_ptr(), s["hu"].numel(), s["mu"].data_ptr(), s["stream"].cuda_stream)
        rc.set_volumes_device([s["vol"]], [s["mu"].data_ptr()], s["dtype"])
        rc.distribute_xforms_among_cam_models(s["poses"])
        rc.compute()
        return {"mu": s["mu"], "drr": s["drr"]}
    if kind == "xray":
        img, cam = xr.proj_preproc(s["raw"], s["cam"])
        return {"image": img, "levels": [xr.downsample_image(img, f) for f in s["f"]]}
    s["m"].compute()
    return s["m"].sim_vals()


# ------------------------------------------------------------------ what a pass cannot do without
def _samples(c, pop):
    """Samples of the step rule inside the body (or, in noisy air, inside the volume) that the detector sees."""
    size, sp = _geometry(c)
    ext = [n * s for n, s in zip(size, sp)]
    px = PANEL / max(c["rows"], c["cols"]) * SOD / SDD
    if c.get("air") == "noisy":
        v = min(ext[0], px * c["cols"]) * ext[1] * min(ext[2], px * c["rows"])
    else:
        v = math.pi / 6 * min(0.86 * ext[0], px * c["cols"]) * 0.68 * ext[1] * min(0.89 * ext[2], px * c["rows"])
    return c["views"] * pop * v / (px * px) / c["step"]


def work(case):
    c, kind = case, case["kind"]
    if kind == "jobs":
        parts = [work(j) for j in _job_cases(c)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "xray":
        n = (c["rows"] - 100) * (c["cols"] - 100)
        out = n * (c["f1"] ** 2 + c["f2"] ** 2)
        # smoothing (9 taps a pass, two passes) and the spline's prefilter (8) and weights (60) per level
        return {"bytes": 4.0 * (c["rows"] * c["cols"] + n + out), "flops": 30.0 * n + 2 * 60.0 * n + 60.0 * out}
    if kind == "images":
        n = c["rows"] * c["cols"]
        return {"bytes": 4.0 * n * (c["n"] + 1) + 4.0 * c["n"], "flops": c["n"] * n * (6.0 if c["metric"] == "ncc" else 40.0)}
    npix, vox = c["rows"] * c["cols"], c["nx"] * c["ny"] * c["nz"]
    drr = 4.0 * npix * c["views"] * c["pop"]
    flops = 24.0 * _samples(c, c["pop"])
    vb = 4 if c["dtype"] == "f32" else 2
    if kind == "admit":
        # HU in, attenuation out, the caster's voxels out
        return {"bytes": vox * (4.0 + 4.0 + vb) + drr, "flops": flops + 4.0 * vox}
    if kind == "render":
        return {"bytes": float(vox * vb) + drr, "flops": flops}
    per_px = {"ncc": 6.0, "grad_ncc": 60.0, "patch_ncc": 40.0, "patch_grad_ncc": 100.0}[c["metric"]]
    return {"bytes": vox * vb + drr + 4.0 * npix * c["views"] + 132.0 * c["pop"], "flops": flops + per_px * npix * c["views"] * c["pop"]}


# ------------------------------------------------------------------ the same results in 64 bits
def _blur_sobel(img):
    """5x5 binomial blur, then the Sobel derivatives, reflected borders; img [n, rows, cols] in double."""
    k = torch.tensor([1.0, 4.0, 6.0, 4.0, 1.0], dtype=torch.float64, device="cuda") / 16.0
    x = F.pad(img[:, None], (2, 2, 2, 2), mode="reflect")
    x = F.pad(F.conv2d(F.conv2d(x, k.view(1, 1, 1, 5)), k.view(1, 1, 5, 1)), (1, 1, 1, 1), mode="reflect")
    d, s = torch.tensor([-1.0, 0.0, 1.0], dtype=torch.float64, device="cuda"), torch.tensor([1.0, 2.0, 1.0], dtype=torch.float64, device="cuda")
    gx = F.conv2d(F.conv2d(x, d.view(1, 1, 1, 3)), s.view(1, 1, 3, 1))[:, 0]
    gy = F.conv2d(F.conv2d(x, s.view(1, 1, 1, 3)), d.view(1, 1, 3, 1))[:, 0]
    return gx, gy


def _ncc64(f, m, mask):
    f, m = f[mask], m[:, mask]
    n = f.numel()
    f, m = f - f.mean(), m - m.mean(1, keepdim=True)
    sd = lambda x: ((x * x).sum(-1) / (n - 1)).sqrt().clamp(min=1e-6)  # noqa: E731
    return 0.5 * (1.0 - (m * f).sum(1) / (n * sd(f) * sd(m)))


def _patch64(f, m, mask, radius, stride):
    """Mask-weighted mean of 1 - ncc over (2 radius + 1)^2 patches (the default options)."""
    d, rows, cols = 2 * radius + 1, f.shape[0], f.shape[1]
    un = lambda x: F.unfold(x[None, None], d, stride=stride)[0]  # noqa: E731  [d * d, patches]
    pf, pm = un(f), un(mask.double())
    n = d * d
    pf = pf - pf.mean(0)
    sf = ((pf * pf).sum(0) / (n - 1)).sqrt().clamp(min=1e-6)
    w = torch.ones(pf.shape[1], dtype=torch.float64, device="cuda")
    if not bool(mask.all()):
        w = pm.mean(0)
        w = w / w.sum()
    keep = w.abs() > 1e-6
    out = []
    for img in m:
        p = un(img)
        p = p - p.mean(0)
        sm = ((p * p).sum(0) / (n - 1)).sqrt().clamp(min=1e-6)
        score = 1.0 - (p * pf * pm).sum(0) / (n * sf * sm)
        out.append((w * score)[keep].sum() / w.sum())
    return torch.stack(out)


def _metric64(metric, f, m, mask, radius=5, stride=1):
    f, m = f.double(), m.double()
    mask = torch.ones_like(f, dtype=torch.bool) if mask is None else torch.from_numpy(mask).cuda().bool()
    pairs = [(f, m)]
    if "grad" in metric:
        (fx, fy), (mx, my) = _blur_sobel(f[None]), _blur_sobel(m)
        pairs = [(fx[0], mx), (fy[0], my)]
    if metric.startswith("patch"):
        return sum(_patch64(a, b, mask, radius, stride) for a, b in pairs) / len(pairs)
    return sum(_ncc64(a, b, mask) for a, b in pairs) / len(pairs)


def _objective64(c, seed):
    size, sp = _geometry(c)
    hu = _hu(size, sp, seed, c["air"])
    vol = _mu64(hu).float().double()
    poses = _poses(size, sp, c["pop"], c["rot"], c["trans"], seed)
    drr = torch.stack([_drr(vol, size, sp, c["rows"], c["cols"], v, p, c["step"]) for v in range(c["views"]) for p in poses])
    fixed = _fixed(hu, size, sp, c, seed)
    mask = _mask(c["rows"], c["cols"], seed) if c["mask"] else None
    sims = sum(_metric64(c["metric"], torch.from_numpy(f).cuda(), drr[v * c["pop"]:(v + 1) * c["pop"]], mask)
               for v, f in enumerate(fixed)) / c["views"]
    return sims.cpu().numpy(), drr


def _gauss_taps(variance, max_error, width):
    """Lindeberg's discrete Gaussian exp(-t) I_k(t), cut where its two-sided sum reaches 1 - max_error, sum 1."""
    def tap(k):
        term = math.exp(-variance) * (0.5 * variance) ** k / math.factorial(k)
        total = term
        for j in range(1, 400):
            term *= 0.25 * variance * variance / (j * (j + k))
            total += term
        return total

    taps = [tap(0), tap(1)]
    while taps[0] + 2 * sum(taps[1:]) < 1.0 - max_error and len(taps) <= width:
        taps.append(tap(len(taps)))
    total = taps[0] + 2 * sum(taps[1:])
    return [t / total for t in taps]


def _smooth64(img, variance):
    taps = _gauss_taps(variance, 0.01, 32)
    r = len(taps) - 1
    k = torch.tensor(taps[:0:-1] + taps, dtype=torch.float64, device="cuda")
    x = F.conv2d(F.pad(img[None, None], (r, r, 0, 0), mode="replicate"), k.view(1, 1, 1, -1))
    return F.conv2d(F.pad(x, (0, 0, r, r), mode="replicate"), k.view(1, 1, -1, 1))[0, 0]


def _prefilter64(c):
    """Cubic B-spline coefficients along dim 0 (mirror boundaries), [n, lines]."""
    z, n = math.sqrt(3.0) - 2.0, c.shape[0]
    c = c * 6.0
    k = torch.arange(n, dtype=torch.float64, device="cuda")
    zk = torch.pow(torch.tensor(abs(z), dtype=torch.float64, device="cuda"), k) * torch.where(k % 2 == 0, 1.0, -1.0)
    c[0] = (zk[:, None] * c).sum(0)  # the mirrored tail is below z^(n - 1)
    for i in range(1, n):
        c[i] += z * c[i - 1]
    c[n - 1] = z / (z * z - 1.0) * (z * c[n - 2] + c[n - 1])
    for i in range(n - 2, -1, -1):
        c[i] = z * (c[i + 1] - c[i])
    return c


def _resample64(c, factor, n_out):
    """Rows of the spline with coefficients c [n, lines] at i / factor."""
    n = c.shape[0]
    x = torch.arange(n_out, dtype=torch.float64, device="cuda") / factor
    i = x.floor()
    t = x - i
    w = [(1 - t) ** 3 / 6, (4 - 6 * t ** 2 + 3 * t ** 3) / 6, (1 + 3 * t + 3 * t ** 2 - 3 * t ** 3) / 6, t ** 3 / 6]
    out = 0.0
    for k in range(4):
        j = (i.long() - 1 + k).abs()
        j = torch.where(j > n - 1, 2 * (n - 1) - j, j)
        out = out + w[k][:, None] * c[j]
    return torch.where((x < n - 0.5)[:, None], out, 0.0)


def _xray64(c, seed):
    raw = torch.from_numpy(_raw_xray(c, seed)).cuda().double()[50:-50, 50:-50]
    i0 = _smooth64(raw, 2.0).max()
    ok = raw > 1e-6
    img = -torch.log(torch.where(ok, raw, raw[ok].min()) / i0)
    levels = []
    for f in (c["f1"], c["f2"]):
        co = _prefilter64(_prefilter64(_smooth64(img, (0.5 / f) ** 2).T.contiguous()).T.contiguous())
        rows, cols = int(img.shape[0] * f + 0.5), int(img.shape[1] * f + 0.5)
        levels.append(_resample64(_resample64(co, f, rows).T.contiguous(), f, cols).T.cpu().numpy())
    return {"image": img.cpu().numpy(), "levels": levels}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("objective", "operators"):
        sims, drr = _objective64(c, seed)
        return {"sims": sims, "drr": drr}
    if kind == "jobs":
        got = [_objective64(j, seed + 1000 * k) for k, j in enumerate(_job_cases(c))]
        return {"sims": [g[0] for g in got], "drr": [g[1] for g in got]}
    if kind == "xray":
        return _xray64(c, seed)
    if kind == "images":
        fixed, mov = _given_images(c, seed)
        mask = _mask(c["rows"], c["cols"], seed) if c["mask"] else None
        return _metric64(c["metric"], fixed, mov, mask, c["radius"], c["stride"]).cpu().numpy()
    size, sp = _geometry(c)
    mu = _mu64(_hu(size, sp, seed, c["air"]))
    vol = mu.float().double()
    pose = _poses(size, sp, 1, c["rot"], c["trans"], seed)[0]
    drr = torch.stack([_drr(vol, size, sp, c["rows"], c["cols"], v, pose, c["step"], c.get("line", "sum")) for v in range(c["views"])])
    return {"mu": mu, "drr": drr} if kind == "admit" else drr.cpu().numpy()
