"""Frames with short sides in launches that fill the GPU, whose units run along strips of columns (the
order itself: test_units.py): the same images as the plain schedule, which has no units."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import kerrtrace_b200 as kt
from kerrtrace_b200 import workloads
from tests.helpers import run_ours

pytestmark = pytest.mark.gpu
KINDS = [(kt.MODE_REF, kt.PREC_FP32), (kt.MODE_SPEC, kt.PREC_FP32), (kt.MODE_SPEC, kt.PREC_MIXED),
         (kt.MODE_SPEC, kt.PREC_FP64)]


def scene(w, h, mode=kt.MODE_REF, prec=kt.PREC_FP32):
    """The t1 view with its longer side in the field of view."""
    base, cam = workloads.scene("t1")
    c = workloads.scaled(base, w, h)
    c.mode, c.precision, c.max_steps = mode, prec, 100
    c.disk_temperature_scale = base.disk_temperature_scale
    if w > h:
        cam.fov_scale *= h / w
    return c, cam


@pytest.mark.parametrize("mode,prec", KINDS)
@pytest.mark.parametrize("size", [(1, 20001), (20001, 1), (9, 9001), (9001, 6), (17, 6001), (501, 213)])
def test_strips_match_plain(cuda, mode, prec, size):
    cfg, cam = scene(*size, mode, prec)
    a, _, _, ctx = run_ours(cuda, cfg, cam, kt.SCHED_PLAIN)
    b, _, _, _ = run_ours(cuda, cfg, cam, kt.SCHED_WAVEFRONT, ctx=ctx)
    ctx.close()
    assert np.all(b[:, 3] == 1.0) and np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("spp", [2, 7])
@pytest.mark.parametrize("size", [(3, 20001), (9001, 5)])
def test_strips_with_several_samples(cuda, size, spp):
    cfg, cam = scene(*size)
    cfg.spp = spp
    a, _, _, ctx = run_ours(cuda, cfg, cam, kt.SCHED_PLAIN)
    b, _, _, _ = run_ours(cuda, cfg, cam, kt.SCHED_WAVEFRONT, ctx=ctx)
    ctx.close()
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("mode,prec", KINDS)
def test_batch_of_strips_and_patches(cuda, mode, prec):
    jobs = [scene(w, h, mode, prec) for w, h in ((1, 9001), (320, 160), (9001, 3), (17, 3001), (1, 1))]
    bufs = [(cuda.full((c.width * c.height, 4), float("nan"), device="cuda"),
             cuda.zeros(2, dtype=cuda.int32, device="cuda")) for c, _ in jobs]
    b = kt.Batch([(c, cam, h.data_ptr(), e.data_ptr()) for (c, cam), (h, e) in zip(jobs, bufs)])
    b.set_tuning(kt.SCHED_WAVEFRONT, blocks_per_sm=4)
    b.trace()
    cuda.cuda.synchronize()
    for (c, cam), (h, _) in zip(jobs, bufs):
        want, _, _, ctx = run_ours(cuda, c, cam, kt.SCHED_PLAIN)
        ctx.close()
        assert np.array_equal(h.cpu().numpy().view(np.uint32), want.view(np.uint32)), (c.width, c.height)
    b.close()


@pytest.mark.parametrize("size,n", [((1, 4001), 3), ((4001, 3), 2), ((17, 2001), 5)])
def test_views_in_strips(cuda, size, n):
    """Every view of one call has the image of a call of its own, which takes patches (one such frame
    is less than the GPU holds)."""
    cfg, cam = scene(*size)
    bb = cuda.tensor(kt.generate_blackbody_lut(cfg.lut_size, cfg.lut_max_temp, cfg.wavelength_start,
                                               cfg.wavelength_end, cfg.wavelength_step), device="cuda")
    disk = cuda.tensor(kt.generate_disk_lut(kt.build_kerr_params(cfg), cfg.disk_outer_radius, cfg.lut_size),
                       device="cuda")

    def trace(cams):
        hdr = cuda.full((len(cams), size[0] * size[1], 4), float("nan"), device="cuda")
        err = cuda.zeros((len(cams), 2), dtype=cuda.int32, device="cuda")
        cuda.cuda.synchronize()
        kt.check(kt.lib().kt_trace_noalloc(C.byref(cfg), (kt.KtCamera * len(cams))(*cams), len(cams),
                                           C.c_void_p(bb.data_ptr()), C.c_void_p(disk.data_ptr()), None,
                                           C.c_void_p(hdr.data_ptr()), C.c_void_p(err.data_ptr())))
        cuda.cuda.synchronize()
        return hdr.cpu().numpy().view(np.uint32)

    r = float(np.linalg.norm(np.array(cam.cam_pos)))
    cams = []
    for v in range(n):
        c = kt.orbit_camera(r, 70.0, 20.0, azimuth_deg=50.0 * v)
        c.fov_scale = cam.fov_scale
        cams.append(c)
    got = trace(cams)
    for v in range(n):
        assert np.array_equal(got[v], trace(cams[v:v + 1])[0]), v


@pytest.mark.parametrize("size", [(1, 20001), (9001, 6), (17, 6001)])
def test_recording_forward_in_strips(cuda, size):
    cfg, view = workloads.c5(64, kt.PREC_FP32)
    cfg.width, cfg.height = size
    n = size[0] * size[1]
    d = kt.Diff(cfg, view)
    hdr = cuda.full((n, 4), float("nan"), device="cuda")
    err = cuda.zeros(2, dtype=cuda.int32, device="cuda")
    d.forward(workloads.C5_START, hdr.data_ptr(), err.data_ptr())
    c, th = cfg.copy(), workloads.C5_START
    c.spin, c.disk_outer_radius = th[0], th[3]
    c.disk_temperature_scale = float(np.float32(view.base_temperature_scale * th[2]))
    cam, _ = kt.diff_orbit_camera(view.observer_r, th[1], view.azimuth_deg, view.fov_deg)
    want, _, _, ctx = run_ours(cuda, c, cam, kt.SCHED_PLAIN)
    ctx.close()
    assert np.array_equal(hdr.cpu().numpy().view(np.uint32), want.view(np.uint32))
    d.close()


@pytest.mark.parametrize("mode,prec", KINDS)
@pytest.mark.parametrize("spin,radius,inclination", [(0.84, 60.0, 20.0), (-0.23, 30.0, 80.0), (-0.01, 120.0, 55.0)])
def test_schedules_agree_as_documented(cuda, mode, prec, spin, radius, inclination):
    """What kt_schedule promises over cameras, spins and kinds: one sample, every schedule of a frame and of a
    batch has the plain image's bits; three samples, both schedules of a batch have them."""
    base, _ = workloads.scene("c2")
    cfg = workloads.scaled(base, 96, 54)
    cfg.spin, cfg.mode, cfg.precision = spin, mode, prec
    cam = kt.orbit_camera(radius, inclination, 30.0, azimuth_deg=100.0)
    n = cfg.width * cfg.height
    for spp in (1, 3):
        cfg.spp = spp
        want, _, _, ctx = run_ours(cuda, cfg, cam, kt.SCHED_PLAIN)
        want = want.view(np.uint32)
        if spp == 1:
            got, _, _, _ = run_ours(cuda, cfg, cam, kt.SCHED_WAVEFRONT, ctx=ctx)
            assert np.array_equal(got.view(np.uint32), want)
        ctx.close()
        hdr, err = cuda.zeros((n, 4), device="cuda"), cuda.zeros(2, dtype=cuda.int32, device="cuda")
        b = kt.Batch([(cfg, cam, hdr.data_ptr(), err.data_ptr())])
        for schedule in (kt.SCHED_PLAIN, kt.SCHED_WAVEFRONT):
            hdr.zero_()
            b.set_tuning(schedule, blocks_per_sm=4)
            b.trace()
            cuda.cuda.synchronize()
            assert np.array_equal(hdr.cpu().numpy().view(np.uint32), want), (spp, schedule)
        b.close()


@pytest.mark.parametrize("size", [(48, 20), (640, 400)])
def test_kept_frozen_rays_in_units(cuda, size):
    """Frozen rays kept to the end of their budget, in launches of one unit per resident warp and of
    more: the plain schedule's image without them."""
    cfg, cam = scene(*size)
    cfg.max_steps = 3000
    want, _, _, ctx = run_ours(cuda, cfg, cam, kt.SCHED_PLAIN)
    for bps in (3, 4):
        ctx.set_tuning(schedule=kt.SCHED_WAVEFRONT, blocks_per_sm=bps, keep_frozen=1)
        got, _, _, _ = run_ours(cuda, cfg, cam, kt.SCHED_AUTO, ctx=ctx)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    ctx.close()
