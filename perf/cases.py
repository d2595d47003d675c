"""Cases that stand for what a program has this library do, with their inputs, one pass of each and
the values that the pass should give.

A case is a dict of plain values.  Its "kind" names the entry points it goes through:

  tables    both lookup tables generated on the device (a host that builds a table per scene)
  frame     one frame through Context: trace, then the post passes
  renderer  two frames in flight through Renderer, back in pinned host memory
  samples   progressive sampling: a frame refined by a few launches
  batch     many renders of different scenes and sizes in one launch
  views     several views of one scene without device allocation
  post      the post passes alone, fused or as the reference's two launches
  fit       one step of the inverse problem: forward, cotangent of the loss, backward

listed() holds the sizes of the repository's own workloads and tests; draw() spreads the same kinds
over their whole ranges, ragged sizes included.  exact() follows each ray with the same method in
double precision (plain torch), so that a result's distance from it is its rounding error.
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

import kerrtrace_b200 as kt

F64 = torch.float64
PRECISION = {"fp32": kt.PREC_FP32, "mixed": kt.PREC_MIXED, "fp64": kt.PREC_FP64}


# ---- the cases ------------------------------------------------------------------------------

def _frame(name, width, height, **more):
    case = {"name": name, "kind": "frame", "width": width, "height": height, "physics": "reference",
            "precision": "fp32", "spp": 1, "tolerance": 1e-6, "octaves": 5, "bloom": 24.0, "spin": 0.998,
            "r_obs": 100.0, "inclination": 85.0, "fov": 25.0, "r_out": 30.0, "shape": "default"}
    case.update(more)
    return case


def listed():
    return [
        # a table set for one scene, as a host makes it when the spin or the temperature range changes
        {"name": "tables_4096", "kind": "tables", "size": 4096, "wl_step": 10.0},
        # the smallest calls: a thumbnail with two samples per pixel, noise and bloom (the parity scene)
        _frame("frame_96x64", 96, 64, spp=2, tolerance=1e-5, octaves=3, bloom=6.0, spin=0.9, r_obs=30.0,
               inclination=75.0, fov=40.0, r_out=25.0),
        # a small accurate frame without noise or bloom (the 256x256 workload, tolerance 1e-8)
        _frame("frame_256_tight", 256, 256, tolerance=1e-8, octaves=0, bloom=0.0, spin=0.9, r_obs=50.0,
               inclination=80.0, fov=30.0, r_out=20.0),
        # the benchmark frame in the launch shape that the autotuner installs for it
        _frame("frame_1080p", 1920, 1080, shape="tuned"),
        # a square frame of the mixed-precision workload
        _frame("frame_mixed_1024", 1024, 1024, physics="stated", precision="mixed", octaves=0, bloom=0.0,
               spin=0.6, r_obs=60.0, inclination=70.0, fov=20.0),
        # the accurate image that the other precisions are judged by
        _frame("frame_fp64_960x540", 960, 540, physics="stated", precision="fp64"),
        # what a host gets out of the box: config.yaml's frame (2100x900, 4 samples, bloom radius 48)
        {"name": "renderer_2100x900", "kind": "renderer", "width": 2100, "height": 900, "spp": 4, "max_steps": 100},
        # the batched workload at half size: 64 renders of 128x128 to 960x540
        {"name": "batch_64", "kind": "batch", "jobs": 64, "side": 960, "shape": "persistent"},
        # several views of one scene for a host that owns all device memory
        {"name": "views_8x480x270", "kind": "views", "width": 480, "height": 270, "views": 8, "octaves": 5},
        # the post passes of a 4K frame
        {"name": "post_4k", "kind": "post", "width": 3840, "height": 2160, "bloom": 24.0, "passes": "fused",
         "physics": "reference"},
        # the inverse problem, in both of its precisions
        {"name": "fit_fp32_512", "kind": "fit", "width": 512, "height": 512, "precision": "fp32", "adjoint": "own"},
        {"name": "fit_fp64_256", "kind": "fit", "width": 256, "height": 256, "precision": "fp64", "adjoint": "own"},
    ]


def draw(rng: random.Random):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["tables", "frame", "frame", "frame", "frame", "renderer", "samples", "batch", "views", "post",
                       "post", "fit", "fit"])
    if kind == "tables":
        return {"kind": kind, "size": log_int(64, 16384), "wl_step": rng.choice([1.0, 5.0, 10.0, 20.0])}
    if kind == "frame":
        physics = rng.choice(["reference", "reference", "stated"])
        precision = rng.choice(["fp32", "mixed", "fp64"]) if physics == "stated" else "fp32"
        top = {"fp32": 1920, "mixed": 1600, "fp64": 960}[precision]
        width = log_int(48, top)
        c = _frame("", width, max(17, int(width * rng.uniform(0.4, 1.1))), physics=physics, precision=precision,
                   spp=rng.choice([1, 1, 2, 4]) if width < 800 else 1, tolerance=rng.choice([1e-5, 1e-6, 1e-6, 1e-7]),
                   octaves=rng.choice([0, 3, 5, 10]), bloom=rng.choice([0.0, 3.0, 6.5, 24.0, 48.0]),
                   spin=round(rng.uniform(0.0, 0.998), 3), r_obs=round(rng.uniform(30.0, 200.0), 1),
                   inclination=round(rng.uniform(5.0, 89.0), 1), fov=round(rng.uniform(10.0, 60.0), 1),
                   r_out=round(rng.uniform(12.0, 50.0), 1), shape=rng.choice(["default", "plain", "tuned"]))
        del c["name"]
        return c
    if kind == "renderer":
        width = log_int(160, 2100)
        return {"kind": kind, "width": width, "height": max(90, int(width * rng.uniform(0.4, 0.8))),
                "spp": rng.choice([1, 2, 4]), "max_steps": rng.choice([100, 400])}
    if kind == "samples":
        width = log_int(80, 800)
        return {"kind": kind, "width": width, "height": max(45, int(width * rng.uniform(0.4, 0.8))),
                "launches": rng.randint(2, 4), "per_launch": rng.randint(1, 3),
                "physics": rng.choice(["reference", "stated"])}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(2, 64), "side": log_int(100, 960),
                "shape": rng.choice(["default", "persistent"])}
    if kind == "views":
        width = log_int(48, 640)
        return {"kind": kind, "width": width, "height": max(27, int(width * rng.uniform(0.4, 0.8))),
                "views": rng.randint(1, 12), "octaves": rng.choice([0, 5])}
    if kind == "post":
        width = log_int(64, 4096)
        return {"kind": kind, "width": width, "height": max(33, min(2304, int(width * rng.uniform(0.4, 1.1)))),
                "bloom": rng.choice([2.0, 6.5, 24.0, 48.0, round(rng.uniform(1.0, 90.0), 1)]),
                "passes": rng.choice(["fused", "two"]), "physics": rng.choice(["reference", "stated"])}
    width = log_int(48, 512)
    precision = rng.choice(["fp32", "fp64"])
    return {"kind": kind, "width": width, "height": max(33, int(width * rng.uniform(0.5, 1.0))),
            "precision": precision, "adjoint": rng.choice(["own", "fp64"]) if precision == "fp32" else "own"}


# ---- scenes: plain numbers -------------------------------------------------------------------

def _isco(a):
    z1 = 1 + (1 - a * a) ** (1 / 3) * ((1 + a) ** (1 / 3) + (1 - a) ** (1 / 3))
    z2 = math.sqrt(3 * a * a + z1 * z1)
    return 3 + z2 - math.sqrt(max((3 - z1) * (3 + z1 + 2 * z2), 0.0))


def _disk_table(spin, mass, r_out, n):
    """f^(1/4) of the Page-Thorne flux factor on n radii from the ISCO to r_out, in double."""
    a, r_in = spin / mass, _isco(spin / mass) * mass
    rn = (r_in + np.arange(n) / (n - 1) * (r_out - r_in)) / mass
    x, x0 = np.sqrt(rn), math.sqrt(r_in / mass)
    base = math.acos(-a) / 3
    roots = [2 * math.cos(base + k) for k in (0.0, -2 * math.pi / 3, 2 * math.pi / 3)]
    total = np.zeros(n)
    for i, xi in enumerate(roots):
        den = xi * (xi - roots[(i + 1) % 3]) * (xi - roots[(i + 2) % 3])
        if den > 0:
            val = (x - xi) / (x0 - xi)
            total += np.where(val > 0, 3 * (xi - a) ** 2 / den * np.log(np.where(val > 0, val, 1.0)), 0.0)
    q = x - x0 - 1.5 * a * np.log(x / x0) - total
    geo = rn * (rn * x - 3 * x + 2 * a)
    f = np.maximum(q / geo, 0.0)
    f[0] = 0.0
    return f ** 0.25


def _blackbody_table(n, max_temp, wl_start, wl_end, wl_step):
    """Linear-sRGB colour of a blackbody on n temperatures from 0 to max_temp, in double."""
    lam, l = [], np.float32(wl_start)
    while not l > np.float32(wl_end):
        lam.append(float(l))
        l = np.float32(l + np.float32(wl_step))
    lam = np.array(lam)

    def lobe(alpha, mu, s1, s2):
        return alpha * np.exp(-0.5 * ((lam - mu) / np.where(lam < mu, s1, s2)) ** 2)

    cmf = np.stack([lobe(1.056, 599.8, 37.9, 31.0) + lobe(0.362, 442.0, 16.0, 26.7) + lobe(-0.065, 501.1, 20.4, 26.2),
                    lobe(0.821, 568.8, 46.9, 40.5) + lobe(0.286, 530.9, 16.3, 31.1),
                    lobe(1.217, 437.0, 11.8, 36.0) + lobe(0.681, 459.0, 26.2, 13.8)], 1)
    t = np.arange(n) / (n - 1) * max_temp
    with np.errstate(divide="ignore", over="ignore"):
        expo = 1.4388e7 / (lam[None, :] * t[:, None])
        inten = np.where(expo > 80.0, 0.0, 1e15 / lam[None, :] ** 5 / np.expm1(expo))
    xyz = inten @ cmf * wl_step
    m = np.array([[3.240454, -1.5371385, -0.4985314], [-0.969266, 1.8760108, 0.041556],
                  [0.0556434, -0.2040259, 1.0572252]])
    return np.concatenate([xyz @ m.T, np.zeros((n, 1))], 1)


def _camera(r_obs, inclination, azimuth, fov, single=True):
    """Orbit camera looking at the hole, as float32 values (or in double)."""
    i, az = math.radians(inclination), math.radians(azimuth)
    pos = (r_obs * math.sin(i) * math.cos(az), r_obs * math.cos(i), r_obs * math.sin(i) * math.sin(az))
    fwd = [-p / r_obs for p in pos]
    rgt = [math.sin(az), 0.0, -math.cos(az)]
    up = [rgt[1] * fwd[2] - rgt[2] * fwd[1], rgt[2] * fwd[0] - rgt[0] * fwd[2], rgt[0] * fwd[1] - rgt[1] * fwd[0]]
    f32 = lambda v: [float(np.float32(x)) if single else x for x in v]  # noqa: E731
    return {"cam_pos": f32(pos), "fwd": f32(fwd), "rgt": f32(rgt), "up": f32(up),
            "fov_scale": f32([math.tan(math.radians(fov) / 2)])[0]}


def _scene(width, height, spin, r_out, *, mass=1.0, spp=1, tolerance=1e-6, octaves=5, bloom=24.0, physics="reference",
           precision="fp32", lut_size=4096, max_steps=20000, max_temp=2e5):
    """Configuration values of the repository's workloads: disk peak at 1e4 K, horizon at 1.01 r_h."""
    r_h = mass + math.sqrt(max(mass * mass - spin * spin, 0.0))
    peak = float(_disk_table(spin, mass, r_out, lut_size).max())
    return {"width": width, "height": height, "spp": spp, "spin": spin, "mass": mass, "tolerance": tolerance,
            "initial_step": 0.1, "max_steps": max_steps, "max_attempts": 3, "escape_radius": 1000.0,
            "horizon_epsilon": 0.01 * r_h, "disk_outer_radius": r_out, "lut_size": lut_size, "lut_max_temp": max_temp,
            "wavelength_start": 380.0, "wavelength_end": 720.0, "wavelength_step": 10.0,
            "transmittance_cutoff": 1e-2, "sky_grid_divisions": 40, "sky_line_thickness": 5e-4, "sky_intensity": 30.0,
            # the flux factor vanishes for some negative spins: no disk emission
            "disk_temperature_scale": 1e4 / peak if peak > 1e-6 else 0.0, "exposure_scale": 3e-3, "noise_enabled": int(octaves > 0),
            "noise_detail": octaves, "noise_scale": 0.1, "noise_strength": 0.6, "noise_winding": 50.0,
            "noise_seed": 42, "bloom_enabled": int(bloom > 0), "bloom_radius": bloom, "bloom_intensity": 0.5,
            "bloom_threshold": 1.0, "mode": kt.MODE_SPEC if physics == "stated" else kt.MODE_REF,
            "precision": PRECISION[precision]}


def _config(values):
    cfg = kt.config_default()
    for k, v in values.items():
        setattr(cfg, k, v)
    return cfg


def _kt_camera(cam):
    c = kt.KtCamera()
    for k in ("cam_pos", "fwd", "rgt", "up"):
        for i in range(3):
            getattr(c, k)[i] = cam[k][i]
    c.fov_scale = cam["fov_scale"]
    return c


def _scenes(case, seed):
    """The renders of a case as (configuration values, camera) pairs; the seed moves the observer
    (and, in a batch, draws each job's scene)."""
    rng = random.Random(seed)
    kind = case["kind"]
    az, di, dr = rng.uniform(0.0, 360.0), rng.uniform(-1.0, 1.0), rng.uniform(0.98, 1.02)
    if kind == "frame":
        v = _scene(case["width"], case["height"], case["spin"], case["r_out"], spp=case["spp"],
                   tolerance=case["tolerance"], octaves=case["octaves"], bloom=case["bloom"], physics=case["physics"],
                   precision=case["precision"])
        return [(v, _camera(case["r_obs"] * dr, min(89.0, max(2.0, case["inclination"] + di)), az, case["fov"]))]
    if kind == "renderer":
        c = kt.config_default()
        v = {n: x for n, x in c.as_dict().items() if n != "block_dim"}
        v.update(width=case["width"], height=case["height"], spp=case["spp"], max_steps=case["max_steps"])
        return [(v, _camera(30.0 * dr, 80.0 + di, az + k, 60.0)) for k in (0.0, 0.5)]
    if kind == "samples":
        v = _scene(case["width"], case["height"], 0.998, 30.0, physics=case["physics"])
        return [(v, _camera(100.0 * dr, 85.0 + di, az, 25.0))]
    if kind == "views":
        v = _scene(case["width"], case["height"], 0.998, 30.0, octaves=case["octaves"])
        return [(v, _camera(100.0 * dr, 85.0 + di, az + 7.0 * k, 25.0)) for k in range(case["views"])]
    out = []
    side = case["side"]
    sizes = [(max(8, side * 2 // 15), max(8, side * 2 // 15)), (max(8, side * 4 // 15), max(8, side * 4 // 15)),
             (max(8, side * 8 // 15), max(8, side * 8 // 15)), (side, max(8, side * 9 // 16))]
    for j in range(case["jobs"]):
        w, h = sizes[j * 4 // case["jobs"]]
        v = _scene(w, h, rng.uniform(-0.99, 0.99), rng.uniform(12.0, 50.0))
        out.append((v, _camera(rng.uniform(30.0, 200.0), rng.uniform(5.0, 89.0), 0.0, 25.0)))
    return out


def _fit_values(case, seed):
    """(configuration values, view values, starting theta, target theta) of the inverse problem."""
    rng = random.Random(seed)
    target = (0.7 + rng.uniform(-0.02, 0.02), 60.0 + rng.uniform(-1.0, 1.0), 1.0, 25.0 + rng.uniform(-0.5, 0.5))
    start = (0.5 + rng.uniform(-0.02, 0.02), 50.0 + rng.uniform(-1.0, 1.0), 0.8, 20.0 + rng.uniform(-0.5, 0.5))
    v = _scene(case["width"], case["height"], 0.7, 25.0, octaves=0, bloom=0.0, physics="stated",
               precision=case["precision"], lut_size=1024, max_temp=1e5)
    v["horizon_epsilon"] = 0.01
    return v, (50.0, 0.0, 30.0, v["disk_temperature_scale"]), start, target


def _tables_values(case, seed):
    rng = random.Random(seed)
    return {"size": case["size"], "max_temp": rng.uniform(2e4, 2e5), "spin": rng.uniform(0.0, 0.99),
            "r_out": rng.uniform(15.0, 50.0), "wl_step": case["wl_step"]}


# ---- inputs and one pass ---------------------------------------------------------------------

def _zeros(n, width, dtype=torch.float32):
    return torch.zeros((n, width) if width > 1 else n, dtype=dtype, device="cuda")


def _hdr_image(width, height, seed):
    """A frame as the trace makes it: a bright ring with a wide range of brightness on black, and
    thin lines of constant brightness."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    y = (torch.arange(height, device="cuda", dtype=torch.float32)[:, None] / height - 0.5) * 3.0
    x = (torch.arange(width, device="cuda", dtype=torch.float32)[None, :] / width - 0.5) * 2.5
    r = torch.sqrt(x * x + 4.0 * y * y)
    ring = ((r > 0.35) & (r < 1.0)).float() * torch.exp(-3.0 * (r - 0.35))
    tex = torch.exp(torch.randn((height, width), generator=g, device="cuda"))
    tint = torch.rand(3, generator=g, device="cuda") + 0.5
    img = torch.zeros((height, width, 4), device="cuda")
    img[..., :3] = (20.0 * ring * tex)[..., None] * tint
    img[:: max(1, height // 20), :, :3] += 0.09
    img[..., 3] = 1.0
    return img.reshape(-1, 4).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    stream = torch.cuda.current_stream().cuda_stream
    s = {"kind": kind, "case": case, "stream": stream}
    if kind == "tables":
        v = _tables_values(case, seed)
        params = kt.build_kerr_params(_config({"spin": v["spin"], "mass": 1.0}))
        s.update(v, params=params, bb=_zeros(v["size"], 4), disk=_zeros(v["size"], 1))
        return s
    if kind == "post":
        v = _scene(case["width"], case["height"], 0.9, 20.0, bloom=case["bloom"], physics=case["physics"], lut_size=64)
        n = case["width"] * case["height"]
        s.update(ctx=kt.Context(_config(v)), hdr=_hdr_image(case["width"], case["height"], seed),
                 bloom=_zeros(n, 4) if case["passes"] == "two" else None, image=_zeros(n, 1, torch.int32))
        return s
    if kind == "fit":
        v, view, start, target = _fit_values(case, seed)
        n = case["width"] * case["height"]
        d = kt.Diff(_config(v), kt.KtDiffView(*view))
        s.update(diff=d, theta=start, hdr=_zeros(n, 4), goal=_zeros(n, 4), err=_zeros(2, 1, torch.int32),
                 grad=_zeros(4, 1, F64))
        d.forward(target, s["goal"].data_ptr(), s["err"].data_ptr(), stream)
        return s
    renders = _scenes(case, seed)
    v0, cam0 = renders[0]
    n = v0["width"] * v0["height"]
    if kind == "frame":
        ctx = kt.Context(_config(v0))
        schedule = None
        if case["shape"] == "plain":
            schedule = kt.SCHED_PLAIN
        elif case["shape"] == "tuned":  # what Context's autotuner installs for the benchmark frame
            ctx.set_tuning(schedule=kt.SCHED_PLAIN, block_x=16, block_y=8,
                           blocks_per_sm=4 if case["precision"] == "fp64" else 6)
            schedule = kt.SCHED_AUTO
        s.update(ctx=ctx, cam=_kt_camera(cam0), schedule=schedule, hdr=_zeros(n, 4), err=_zeros(2, 1, torch.int32),
                 image=_zeros(n, 1, torch.int32))
    elif kind == "renderer":
        s.update(renderer=kt.Renderer(_config(v0)),
                 cams=[(c["cam_pos"], c["fwd"], c["rgt"], c["up"], c["fov_scale"]) for _, c in renders])
    elif kind == "samples":
        s.update(ctx=kt.Context(_config(v0)), cam=_kt_camera(cam0), accum=_zeros(n, 4), hdr=_zeros(n, 4),
                 err=_zeros(2, 1, torch.int32))
    elif kind == "views":
        bb = torch.from_numpy(kt.generate_blackbody_lut(v0["lut_size"], v0["lut_max_temp"], v0["wavelength_start"],
                                                        v0["wavelength_end"], v0["wavelength_step"])).cuda()
        cfg = _config(v0)
        disk = torch.from_numpy(kt.generate_disk_lut(kt.build_kerr_params(cfg), cfg.disk_outer_radius,
                                                     cfg.lut_size)).cuda()
        cams = (kt.KtCamera * len(renders))(*[_kt_camera(c) for _, c in renders])
        s.update(cfg=cfg, cams=cams, bb=bb, disk=disk, hdr=_zeros(n * len(renders), 4),
                 err=_zeros(2 * len(renders), 1, torch.int32))
    else:
        counts = [v["width"] * v["height"] for v, _ in renders]
        hdr, err = _zeros(sum(counts), 4), _zeros(2 * len(renders), 1, torch.int32)
        jobs, at = [], 0
        for j, (v, cam) in enumerate(renders):
            jobs.append((_config(v), _kt_camera(cam), hdr.data_ptr() + 16 * at, err.data_ptr() + 8 * j))
            at += counts[j]
        batch = kt.Batch(jobs)
        if case["shape"] == "persistent":  # what Batch's autotuner installs for the batched workload
            batch.set_tuning(schedule=kt.SCHED_WAVEFRONT, blocks_per_sm=5)
        s.update(batch=batch, hdr=hdr, err=err)
    return s


class _Frame(np.ndarray):
    """A frame in a renderer's pinned memory, which lives as long as the frame is held."""


def run(s):
    kind, case, stream = s["kind"], s["case"], s["stream"]
    if kind == "tables":
        kt.generate_blackbody_lut_device(s["size"], s["max_temp"], 380.0, 720.0, s["wl_step"], s["bb"].data_ptr(), stream)
        kt.generate_disk_lut_device(s["params"], s["r_out"], s["size"], s["disk"].data_ptr(), stream)
        return {"bb": s["bb"], "disk": s["disk"]}
    if kind == "post":
        if case["passes"] == "fused":
            s["ctx"].post_fused(s["hdr"].data_ptr(), s["image"].data_ptr(), stream)
            return {"image": s["image"]}
        s["ctx"].bloom_horizontal(s["hdr"].data_ptr(), s["bloom"].data_ptr(), stream)
        s["ctx"].post_process(s["hdr"].data_ptr(), s["bloom"].data_ptr(), s["image"].data_ptr(), stream)
        return {"bloom": s["bloom"], "image": s["image"]}
    if kind == "frame":
        hdr, err = s["hdr"].data_ptr(), s["err"].data_ptr()
        if s["schedule"] is None:
            s["ctx"].trace(s["cam"], hdr, err, stream)
        else:
            s["ctx"].trace(s["cam"], hdr, err, stream, s["schedule"])
        s["ctx"].post_fused(hdr, s["image"].data_ptr(), stream)
        return {"hdr": s["hdr"], "err": s["err"], "image": s["image"]}
    if kind == "renderer":
        r, images = s["renderer"], []
        for cam in s["cams"]:
            r.submit_render(*cam)
        r.wait()
        for _ in s["cams"]:
            index, image = r.ready_frame()
            images.append(image.view(_Frame))
            images[-1].renderer = r
            r.finish_frame(index)
        return {"images": images}
    if kind == "samples":
        for k in range(case["launches"]):
            s["ctx"].trace_progressive(s["cam"], k * case["per_launch"], case["per_launch"], s["accum"].data_ptr(),
                                       s["hdr"].data_ptr(), s["err"].data_ptr(), stream)
        return {"accum": s["accum"], "hdr": s["hdr"], "err": s["err"]}
    if kind == "views":
        vp = ctypes.c_void_p
        kt.check(kt.lib().kt_trace_noalloc(ctypes.byref(s["cfg"]), s["cams"], len(s["cams"]), vp(s["bb"].data_ptr()),
                                           vp(s["disk"].data_ptr()), vp(stream), vp(s["hdr"].data_ptr()),
                                           vp(s["err"].data_ptr())))
        return {"hdr": s["hdr"], "err": s["err"]}
    if kind == "batch":
        s["batch"].trace(stream)
        return {"hdr": s["hdr"], "err": s["err"]}
    d = s["diff"]
    d.forward(s["theta"], s["hdr"].data_ptr(), s["err"].data_ptr(), stream)
    cotangent = s["hdr"] - s["goal"]
    if case["adjoint"] == "fp64":
        d.backward_fp64(cotangent.data_ptr(), s["grad"].data_ptr(), stream)
    else:
        d.backward(cotangent.data_ptr(), s["grad"].data_ptr(), stream)
    # an FP32 object's parameters are float32 numbers of the caller's program, and so is their gradient
    single = case["precision"] == "fp32" and case["adjoint"] == "own"
    return {"hdr": s["hdr"], "grad": s["grad"].float() if single else s["grad"]}


def work(case):
    """Bytes: outputs written and inputs read once.  Flops of a trace: about 30 attempts per ray at
    tolerance 1e-6 (order 5: 1.58 times as many per decade), 6 right-hand sides of 160 and 371 of
    stage arithmetic each."""
    kind = case["kind"]
    if kind == "tables":
        return {"bytes": 20 * case["size"], "flops": case["size"] * (340.0 / case["wl_step"] + 1) * 20}
    if kind == "post":
        n = case["width"] * case["height"]
        out = 4 if case["passes"] == "fused" else 20
        return {"bytes": n * (16 + out), "flops": n * 2 * (2 * math.ceil(case["bloom"]) + 1) * 6}
    attempt = 6 * 160 + 371
    if kind == "batch":
        rays = sum(v["width"] * v["height"] for v, _ in _scenes(case, 0))
        return {"bytes": 16 * rays, "flops": 30.0 * attempt * rays}
    n = case["width"] * case["height"]
    if kind == "fit":
        return {"bytes": 3 * 16 * n, "flops": 28.0 * attempt * n * 3.5}
    rays, out = n * case.get("spp", 1), 20
    if kind == "samples":
        rays, out = n * case["launches"] * case["per_launch"], 48
    elif kind == "views":
        rays, n, out = n * case["views"], n * case["views"], 16
    elif kind == "renderer":
        rays, n = 2 * rays, 2 * n
    per_ray = 30.0 * (1e-6 / case.get("tolerance", 1e-6)) ** 0.2
    return {"bytes": out * n, "flops": per_ray * attempt * rays}


# ---- the same results in double precision, plain torch ---------------------------------------

def _pcg(state):
    """PCG32 output of 64-bit states (int64 tensors, wrapping arithmetic, logical shifts)."""
    x = state * 6364136223846793005 + 1442695040888963407
    low = lambda v, k: (v >> k) & ((1 << (64 - k)) - 1)  # noqa: E731
    xs = low(low(x, 18) ^ x, 27) & 0xFFFFFFFF
    rot = low(x, 59)
    return ((xs >> rot) | (xs << ((32 - rot) & 31))) & 0xFFFFFFFF


def _signed(v):
    return v - (1 << 64) if v >= 1 << 63 else v


def _directions(v, cam, sample, centre):
    w, h = v["width"], v["height"]
    p = torch.arange(w * h, device="cuda", dtype=torch.int64)
    px, py = (p % w).to(F64), (p // w).to(F64)
    if centre:
        jx = jy = 0.5
    else:
        key = (p << 32) | sample
        jx = _pcg(key).to(F64) * 2.0 ** -32
        jy = _pcg(key ^ _signed(0xDA3E39CB94B95BDB)).to(F64) * 2.0 ** -32
    u = ((px + jx) * 2.0 / w - 1.0) * (w / h) * cam["fov_scale"]
    t = (1.0 - (py + jy) * 2.0 / h) * cam["fov_scale"]
    return torch.stack([u * cam["rgt"][c] + t * cam["up"][c] + cam["fwd"][c] for c in range(3)])


def _radius(x, y, z, aa):
    u = x * x + y * y + z * z - aa
    return torch.sqrt(0.5 * (u + torch.sqrt(u * u + 4 * aa * y * y)))


def _rhs(s, pt, a, m, stated):
    """Hamilton's equations of H = (p.p - pt^2)/2 - Hk (l.p - pt)^2; the reference's own form of
    dr/dy where `stated` is false."""
    x, y, z, px, py, pz = s
    aa = a * a
    u = x * x + y * y + z * z - aa
    inv_s = torch.rsqrt(u * u + 4 * aa * y * y)
    r2 = 0.5 * (u + 1 / inv_s)
    r = torch.sqrt(r2)
    g = (1 + u * inv_s) / (2 * r)
    gy = (1 + (u + 2 * aa) * inv_s) / (2 * r) if stated else (1 + 0.5 * (u + 4 * aa) * inv_s) / (2 * r)
    den = r2 + aa
    nx, nz = r * x - a * z, r * z + a * x
    lx, ly, lz = nx / den, y / r, nz / den
    den_h = r2 * r2 + aa * y * y
    hk = m * r2 * r / den_h
    lp = lx * px + ly * py + lz * pz - pt
    w = 2 * hk * lp
    c = (x * px + z * pz - 2 * r * (nx * px + nz * pz) / den) / den - py * y / r2
    q = m * r2 * (3 * aa * y * y - r2 * r2) / den_h ** 2 * lp * lp + w * c
    return torch.stack([px - w * lx, py - w * ly, pz - w * lz, x * g * q + w * (r * px + a * pz) / den,
                        y * gy * q - 2 * m * aa * y * r2 * r / den_h ** 2 * lp * lp + w * py / r,
                        z * g * q + w * (r * pz - a * px) / den])


_A = [[1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
      [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
      [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
      [35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]]
_E = [35 / 384 - 5179 / 57600, 0.0, 500 / 1113 - 7571 / 16695, 125 / 192 - 393 / 640, -2187 / 6784 + 92097 / 339200,
      11 / 84 - 187 / 2100, -1 / 40]
_D = [-12715105075 / 11282082432, 0.0, 87487479700 / 32700410799, -10690763975 / 1880347072,
      701980252875 / 199316789632, -1453857185 / 822651844, 69997945 / 29380423]


def _combine(weights, ks):
    out = weights[0] * ks[0]
    for w, k in zip(weights[1:], ks[1:]):
        if w:
            out = out + w * k
    return out


def _dense(y0, y1, ks, h, t, slope=False):
    q2, q3 = y1 - y0, y0 + h * ks[0] - y1
    q4 = 2 * (y1 - y0) - h * (ks[0] + ks[6])
    q5 = h * _combine(_D, ks)
    if slope:
        return q2 + q3 - 2 * t * (q3 - q4 - q5) - 3 * t * t * (q4 + 2 * q5) + 4 * t ** 3 * q5
    return y0 + t * (q2 + q3) - t * t * (q3 - q4 - q5) - t ** 3 * (q4 + 2 * q5) + t ** 4 * q5


def _lerp(table, x):
    n = table.shape[0]
    fl = torch.floor(x)
    i0 = fl.clamp(0, n - 1).long()
    i1 = (fl + 1).clamp(0, n - 1).long()
    w = (x - fl)
    if table.dim() == 2:
        w = w[:, None]
    return table[i0] + w * (table[i1] - table[i0])


def _fbm(u, v, octaves, seed):
    def gradient(ix, iy):
        key = ((ix & 0xFFFFFFFF) << 32) | (iy & 0xFFFFFFFF)
        ang = _pcg(key ^ seed).to(F64) * (2 * math.pi * 2.0 ** -32)
        return torch.cos(ang), torch.sin(ang)

    total, amp, amps = torch.zeros_like(u), 1.0, 0.0
    for _ in range(octaves):
        ix, iy = torch.floor(u).long(), torch.floor(v).long()
        fx, fy = u - ix, v - iy
        n = []
        for dy in (0, 1):
            for dx in (0, 1):
                gx, gy = gradient(ix + dx, iy + dy)
                n.append(gx * (fx - dx) + gy * (fy - dy))
        su, sv = (t ** 3 * (t * (t * 6 - 15) + 10) for t in (fx, fy))
        lo, hi = n[0] + su * (n[1] - n[0]), n[2] + su * (n[3] - n[2])
        total = total + amp * (lo + sv * (hi - lo))
        amps += amp
        amp *= 0.5
        u, v = 2 * u, 2 * v
    return total / amps * 0.5 + 0.5


class _Tracer:
    """The renderer's integrator and shading in double, on all rays of a scene at once."""

    def __init__(self, v):
        self.v, self.stated = v, v["mode"] == kt.MODE_SPEC
        self.a, self.m = float(v["spin"]), float(v["mass"])
        self.r_in, self.r_out = _isco(self.a / self.m) * self.m, v["disk_outer_radius"]
        self.horizon = self.m + math.sqrt(max(self.m ** 2 - self.a ** 2, 0.0)) + round(v["horizon_epsilon"], 10)
        self.disk = torch.from_numpy(_disk_table(self.a, self.m, self.r_out, v["lut_size"])).cuda()
        self.bb = torch.from_numpy(_blackbody_table(v["lut_size"], v["lut_max_temp"], v["wavelength_start"],
                                                    v["wavelength_end"], v["wavelength_step"])[:, :3]).cuda()

    def tolerance(self, r, y):
        hk = self.m * r ** 3 / (r ** 4 + self.a ** 2 * y * y)
        t = ((hk - 0.05) / 0.25).clamp(0.0, 1.0)
        return self.v["tolerance"] * (5.0 - (4.0 if self.stated else 5.0) * t)

    def shade(self, hit, pt, kt_):
        """(colour, opacity) of disk-plane hits; opacity 0 where nothing is shaded."""
        v, a, m = self.v, self.a, self.m
        x, z, px, pz = hit[0], hit[2], hit[3], hit[5]
        r = _radius(x, torch.zeros_like(x), z, a * a)
        rs = torch.sqrt(r)
        disc = 1 - 3 * m / r + 2 * a * math.sqrt(m) / (r * rs)
        on = (r >= self.r_in) & (r <= self.r_out) & (disc > 0)
        omega = -math.sqrt(m) / (r * rs + a * math.sqrt(m))
        lx, lz = (r * x - a * z) / (r * r + a * a), (r * z + a * x) / (r * r + a * a)
        spin_l = (z * px - x * pz) + 2 * m / r * (lx * z - lz * x) * (lx * px + lz * pz + kt_)
        g = torch.sqrt(disc.clamp(min=0)) / (1 + omega * spin_l / pt)
        u = (r - self.r_in) / (self.r_out - self.r_in)
        temp = v["disk_temperature_scale"] * _lerp(self.disk, u * v["lut_size"] - 0.5) * g
        if v["noise_enabled"] and v["noise_detail"] > 0 and v["noise_strength"] != 0.0:
            phi = torch.atan2(r * x - a * z, r * z + a * x)
            phase = phi + v["noise_winding"] / (a + torch.sqrt(r ** 3 / m))
            n = _fbm(r * torch.cos(phase) * v["noise_scale"], r * torch.sin(phase) * v["noise_scale"],
                     v["noise_detail"], v["noise_seed"] if self.stated else 0)
            temp = temp * (1 + v["noise_strength"] * (n - 0.5))
        on &= torch.isfinite(temp) & (temp > 0)
        temp = torch.where(on, temp, torch.ones_like(temp))
        c = _lerp(self.bb, (temp / v["lut_max_temp"]).clamp(max=1.0) * (v["lut_size"] - 1))
        on &= temp <= v["lut_max_temp"]
        luma = (c @ torch.tensor([0.2126, 0.7152, 0.0722], dtype=F64, device="cuda")) / v["wavelength_step"]
        return c, torch.where(on, 1 - torch.exp(-0.5 * luma), torch.zeros_like(luma))

    def sky(self, s, pt):
        d = _rhs(s, pt, self.a, self.m, self.stated)[:3]
        d = d / torch.linalg.vector_norm(d, dim=0)
        lon, lat = torch.atan2(d[2], d[0]).abs(), torch.asin(d[1]).abs()
        gap, thick = math.pi / self.v["sky_grid_divisions"], self.v["sky_line_thickness"]
        line = lat < 3 * thick
        for ang in (lon, lat):
            m = torch.fmod(ang, gap)
            line = line | (m < thick) | (m > gap - thick)
        return line.to(F64) * self.v["sky_intensity"]

    def trace(self, pos, d, limit=4000):
        """Colours (N, 3) of rays from `pos` (3,) or (3, N) along d (3, N)."""
        v, a, m = self.v, self.a, self.m
        n = d.shape[1]
        pos = pos if pos.dim() == 2 else pos[:, None].expand(3, n)
        d = d / torch.linalg.vector_norm(d, dim=0)
        x, y, z = pos
        r = _radius(x, y, z, a * a)
        l = torch.stack([(r * x - a * z) / (r * r + a * a), y / r, (r * z + a * x) / (r * r + a * a)])
        hk = m * r ** 3 / (r ** 4 + a * a * y * y)
        ln = (l * d).sum(0)
        g_tt, g_tn, g_nn = 2 * hk - 1, 2 * hk * ln, 1 + 2 * hk * ln * ln
        kt_ = (-g_tn - torch.sqrt(g_tn * g_tn - g_tt * g_nn)) / g_tt
        pt = g_tt * kt_ + g_tn
        out = torch.zeros((n, 3), dtype=F64, device="cuda")
        at = torch.arange(n, device="cuda")
        s = torch.cat([pos, d + 2 * hk * l * (kt_ + ln)])
        h = torch.full((n,), float(np.float32(round(v["initial_step"], 10))), dtype=F64, device="cuda")
        tol, k1 = self.tolerance(r, y), _rhs(s, pt, a, m, self.stated)
        tau = torch.ones(n, dtype=F64, device="cuda")
        tried, steps = torch.zeros(n, dtype=torch.int32, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
        live = torch.ones(n, dtype=torch.bool, device="cuda")
        for it in range(limit):
            if it % 8 == 0:
                keep = live.nonzero()[:, 0]
                if not len(keep):
                    break
                if len(keep) < 0.9 * len(live) or len(keep) < len(live) and it % 64 == 0:
                    at, s, k1 = at[keep], s[:, keep], k1[:, keep]
                    pt, kt_, h, tol, tau = pt[keep], kt_[keep], h[keep], tol[keep], tau[keep]
                    tried, steps, live = tried[keep], steps[keep], live[keep]
            ks = [k1]
            for row in _A:
                nx = s + h * _combine(row, ks)
                ks.append(_rhs(nx, pt, a, m, self.stated))
            e = (h * _combine(_E, ks)).abs() / (tol * s.abs().clamp(min=1.0))
            err = e[0]
            for c in range(1, 6):
                err = torch.fmax(err, e[c])
            ok = err <= 1
            tried = tried + 1
            commit = live & (ok | (tried >= v["max_attempts"]))
            step_h, h = h, torch.where(live, h * 0.9 * err ** -0.2, h)
            prev = s
            s = torch.where(commit, nx, s)
            tried = torch.where(commit, torch.zeros_like(tried), tried)
            k1 = torch.where(commit, ks[6], k1)
            r = _radius(s[0], s[1], s[2], a * a)
            live = live & ~(commit & (torch.isnan(s[1]) | (r < self.horizon)))
            commit = commit & live
            cross = commit & (((prev[1] < 0) & (s[1] >= 0)) | ((prev[1] > 0) & (s[1] <= 0)))
            i = cross.nonzero()[:, 0]
            if len(i):
                y0, y1, hi = prev[:, i], s[:, i], step_h[i]
                ki = [k[:, i] for k in ks]
                t = (y0[1] / (y0[1] - y1[1])).clamp(0, 1)
                if self.stated:
                    k_y = [k[1] for k in ki]
                    lo, up = torch.zeros_like(t), torch.ones_like(t)
                    for _ in range(50):
                        f = _dense(y0[1], y1[1], k_y, hi, t)
                        same = (f < 0) == (y0[1] < 0)
                        lo, up = torch.where(same, t, lo), torch.where(same, up, t)
                        tn = t - f / _dense(y0[1], y1[1], k_y, hi, t, slope=True)
                        t = torch.where((tn >= lo) & (tn <= up), tn, 0.5 * (lo + up))
                colour, alpha = self.shade(_dense(y0, y1, ki, hi, t), pt[i], kt_[i])
                out[at[i]] += colour * (alpha * tau[i])[:, None]
                tau[i] *= 1 - alpha
            gone = commit & (r > v["escape_radius"])
            i = gone.nonzero()[:, 0]
            if len(i):
                out[at[i]] += (self.sky(s[:, i], pt[i]) * tau[i])[:, None]
            steps = steps + commit.int()
            live = live & ~gone & ~(commit & ((steps >= v["max_steps"]) | (tau <= v["transmittance_cutoff"])))
            tol = torch.where(commit, self.tolerance(r, s[1]), tol)
        return out


def _image(v, cams, samples, centre):
    """Sum of the samples' colours for every camera, (cameras x pixels, 3)."""
    n, k = v["width"] * v["height"], len(samples)
    d = torch.cat([_directions(v, c, i, centre) for i in samples for c in cams], 1)
    pos = torch.cat([torch.tensor(c["cam_pos"], dtype=F64, device="cuda")[:, None].expand(3, n) for c in cams], 1)
    return _Tracer(v).trace(pos.repeat(1, k), d).reshape(k, len(cams) * n, 3).sum(0)


def _rgba(rgb, alpha=1.0):
    return torch.cat([rgb, torch.full_like(rgb[:, :1], alpha)], 1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "tables":
        v = {k: float(np.float32(x)) if k in ("max_temp", "r_out", "spin") else x
             for k, x in _tables_values(case, seed).items()}
        return {"bb": torch.from_numpy(_blackbody_table(v["size"], v["max_temp"], 380.0, 720.0, v["wl_step"])),
                "disk": torch.from_numpy(_disk_table(v["spin"], 1.0, v["r_out"], v["size"]))}
    if kind == "post":
        if case["passes"] == "fused" or case["physics"] == "stated":
            return {"bloom": None, "image": None} if case["passes"] == "two" else None
        img = _hdr_image(case["width"], case["height"], seed).reshape(case["height"], case["width"], 4)[..., :3].to(F64)
        n = math.ceil(case["bloom"])
        w = torch.exp(-torch.arange(-n, n + 1, dtype=F64, device="cuda") ** 2 / (2 * (case["bloom"] / 3) ** 2))
        total, norm = torch.zeros_like(img), torch.zeros(case["width"], dtype=F64, device="cuda")
        for k in range(-n, n + 1):
            a, b = max(0, -k), min(case["width"], case["width"] - k)
            if a < b:
                total[:, a:b] += w[k + n] * img[:, a + k:b + k]
                norm[a:b] += w[k + n]
        return {"bloom": _rgba((total / norm[:, None]).reshape(-1, 3), 0.0), "image": None}
    if kind in ("renderer", "batch"):  # whole numbers; 64 scenes take minutes
        return None
    if kind == "fit":
        v, view, theta, _ = _fit_values(case, seed)
        v.update(spin=theta[0], disk_outer_radius=theta[3], disk_temperature_scale=view[3] * theta[2])
        cam = _camera(view[0], theta[1], view[1], view[2], single=case["precision"] == "fp32")
        rgb = _image(v, [cam], [0], True) * v["exposure_scale"]
        return {"hdr": _rgba(rgb), "grad": None}
    renders = _scenes(case, seed)
    v, cams = renders[0][0], [c for _, c in renders]
    if kind == "samples":
        count = case["launches"] * case["per_launch"]
        if v["width"] * v["height"] * count > 400_000:
            return None
        rgb = _image(v, cams, range(count), False)
        return {"accum": _rgba(rgb, float(count)), "hdr": _rgba(rgb * v["exposure_scale"] / count), "err": None}
    rgb = _image(v, cams, range(v["spp"]), v["mode"] == kt.MODE_SPEC and v["spp"] == 1)
    out = {"hdr": _rgba(rgb * v["exposure_scale"] / v["spp"]), "err": None}
    return dict(out, image=None) if kind == "frame" else out
