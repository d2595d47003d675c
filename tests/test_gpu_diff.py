"""Differentiable trace (kt_diff_*) on the GPU: the recorded forward is the renderer's image,
the frozen-step replay reproduces it, and the discrete adjoint matches central differences of
the frozen-step model (FP64, double images) in total and pixel by pixel; the FP32 adjoint tracks
the FP64 one.  Scene: the inverse-problem workload at 64x64, at its starting parameters."""
from __future__ import annotations

import numpy as np
import pytest

import kerrtrace_b200 as kt
from kerrtrace_b200 import workloads

pytestmark = pytest.mark.gpu

SIZE = 64
THETA = list(workloads.C5_START)
EPS = [1e-5, 1e-4, 1e-5, 1e-4]  # spin, inclination (deg), temperature scale, r_out
NAMES = ["spin", "inclination", "temperature scale", "r_out"]


def make(prec):
    cfg, view = workloads.c5(SIZE, prec)
    return cfg, view, kt.Diff(cfg, view)


def forward(torch, d, theta):
    n = SIZE * SIZE
    hdr = torch.zeros((n, 4), device="cuda")
    err = torch.zeros(2, dtype=torch.int32, device="cuda")
    d.forward(theta, hdr.data_ptr(), err.data_ptr())
    torch.cuda.synchronize()
    assert int(err[0]) == 0
    return hdr


def replay(torch, d, theta):
    n = SIZE * SIZE
    hdr = torch.zeros((n, 4), device="cuda")
    h64 = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    flags = torch.zeros(n, dtype=torch.int32, device="cuda")
    err = torch.zeros(2, dtype=torch.int32, device="cuda")
    d.replay(theta, hdr.data_ptr(), flags.data_ptr(), err.data_ptr(), hdr64_ptr=h64.data_ptr())
    torch.cuda.synchronize()
    return hdr, h64, flags.bool()


def backward(torch, d, w):
    g = torch.zeros(4, dtype=torch.float64, device="cuda")
    d.backward(w.data_ptr(), g.data_ptr())
    torch.cuda.synchronize()
    return g.cpu().numpy()


def replay_fp64(torch, d, theta):
    """The recorded step sequence replayed in double arithmetic (FP32 records for an FP32 object)."""
    n = SIZE * SIZE
    hdr = torch.zeros((n, 4), device="cuda")
    h64 = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    flags = torch.zeros(n, dtype=torch.int32, device="cuda")
    err = torch.zeros(2, dtype=torch.int32, device="cuda")
    d.replay_fp64(theta, h64.data_ptr(), flags.data_ptr(), err.data_ptr(), hdr.data_ptr())
    torch.cuda.synchronize()
    return hdr, h64, flags.bool()


def central_differences(torch, d, replay_fn=None):
    """Richardson-extrapolated central differences per pixel and parameter, and the mask of
    pixels they cannot resolve: event flips under the perturbation, and pixels whose
    differences at eps and eps/2 disagree (a LUT cell edge or a sky-line edge inside the step)."""
    replay_fn = replay_fn or replay
    n = SIZE * SIZE
    mask = torch.zeros(n, dtype=torch.bool, device="cuda")
    fd = []
    for j in range(4):
        img = {}
        for sgn in (1, -1):
            for k in (1, 2):
                t2 = list(THETA)
                t2[j] += sgn * EPS[j] / k
                _, h64, flags = replay_fn(torch, d, t2)
                img[(sgn, k)] = h64
                mask |= flags
        f1 = (img[(1, 1)] - img[(-1, 1)]) / (2 * EPS[j])
        f2 = (img[(1, 2)] - img[(-1, 2)]) / EPS[j]
        mask |= ((f1 - f2).abs() > 1e-3 * f2.abs() + 1e-7 * f2.abs().max()).any(dim=1)
        fd.append((4 * f2 - f1) / 3)
    return fd, mask


def test_record_is_the_renderer_image_and_replay_reproduces_it(cuda):
    for prec in (kt.PREC_FP32, kt.PREC_FP64):
        cfg, view, d = make(prec)
        hdr = forward(cuda, d, THETA)
        h2, _, flags = replay(cuda, d, THETA)
        assert cuda.equal(h2.view(cuda.int32), hdr.view(cuda.int32))
        assert not bool(flags.any())
        info = d.info()
        assert info.overflow_rays == 0 and 0 < info.segments_used <= info.segments_capacity
        if prec == kt.PREC_FP32:
            c = cfg.copy()
            c.spin, c.disk_outer_radius = THETA[0], THETA[3]
            c.disk_temperature_scale = view.base_temperature_scale * THETA[2]
            cam, _ = kt.diff_orbit_camera(view.observer_r, THETA[1], view.azimuth_deg, view.fov_deg)
            ctx = kt.Context(c)
            h3 = cuda.zeros_like(hdr)
            err = cuda.zeros(2, dtype=cuda.int32, device="cuda")
            ctx.trace(cam, h3.data_ptr(), err.data_ptr(), 0, kt.SCHED_PLAIN)
            cuda.cuda.synchronize()
            assert cuda.equal(h3.view(cuda.int32), hdr.view(cuda.int32))
        d.close()


def test_fp64_adjoint_matches_central_differences(cuda):
    _, _, d = make(kt.PREC_FP64)
    hdr = forward(cuda, d, THETA)
    fd, mask = central_differences(cuda, d)
    lit = hdr[:, :3].sum(1) > 0
    assert int(mask.sum()) <= 0.02 * int(lit.sum())
    n = SIZE * SIZE
    rng = np.random.default_rng(1)
    w = cuda.tensor((rng.standard_normal((n, 4)) + 1.0).astype(np.float32), device="cuda")
    w[:, 3] = 0
    w[mask] = 0
    g = backward(cuda, d, w)
    for j in range(4):
        ref = float((fd[j] * w[:, :3].double()).sum())
        assert abs(g[j] - ref) <= 1e-4 * abs(ref), (NAMES[j], g[j], ref)
    # pixel by pixel (one-hot cotangents)
    cand = np.flatnonzero((lit & ~mask).cpu().numpy())
    pick = np.random.default_rng(2).choice(cand, size=min(40, len(cand)), replace=False)
    rel = [[] for _ in range(4)]
    for p in pick:
        e = cuda.zeros((n, 4), device="cuda")
        e[p, :3] = 1.0
        gp = backward(cuda, d, e)
        for j in range(4):
            f = float(fd[j][p].sum())
            rel[j].append(abs(gp[j] - f) / (abs(f) + 1e-6 * float(fd[j].sum(1).abs().max())))
    for j in range(4):
        assert np.median(rel[j]) < 1e-6 and np.max(rel[j]) < 1e-3, (NAMES[j], np.median(rel[j]), np.max(rel[j]))
    d.close()


def test_fp32_adjoint_matches_central_differences_of_its_model(cuda):
    """The FP32 adjoint differentiates the frozen-step model of the FP32 records.  Replayed in
    double arithmetic (kt_diff_replay_fp64), that model's central differences carry no float
    rounding of the images; the FP32 adjoint of the loss matches them to 1e-4 in spin,
    inclination and temperature scale.  The r_out derivative is a second-order remainder: moving
    r_out moves the disk table's nodes and, at a fixed hit radius, the fetch coordinate, and the two
    cancel to about 1/lut_size of either; the float rounding of the FP32 hit state is amplified by
    that much, so r_out is held to 2e-3 (measured: 3.5e-4 here, 6.9e-4 at 512^2; the FP64
    adjoint meets 1e-4 in all four)."""
    _, _, d = make(kt.PREC_FP32)
    hdr = forward(cuda, d, THETA)
    h0, h64, flags = replay_fp64(cuda, d, THETA)
    assert not bool(flags.any())
    # the FP64 replay of the FP32 records differs from the FP32 image by the rounding the float
    # trajectory accumulates (about 1e-4 of the image maximum)
    assert float((h64 - hdr[:, :3].double()).abs().max()) <= 3e-4 * float(hdr[:, :3].abs().max())
    fd, mask = central_differences(cuda, d, replay_fp64)
    lit = hdr[:, :3].sum(1) > 0
    assert int(mask.sum()) <= 0.02 * int(lit.sum())
    n = SIZE * SIZE
    rng = np.random.default_rng(1)
    w = cuda.tensor((rng.standard_normal((n, 4)) + 1.0).astype(np.float32), device="cuda")
    w[:, 3] = 0
    w[mask] = 0
    g = backward(cuda, d, w)
    for j in range(4):
        ref = float((fd[j] * w[:, :3].double()).sum())
        print(NAMES[j], g[j], ref, abs(g[j] - ref) / abs(ref))
        assert abs(g[j] - ref) <= (2e-3 if j == 3 else 1e-4) * abs(ref), (NAMES[j], g[j], ref)
    d.close()


def backward_fp64(torch, d, w):
    g = torch.zeros(4, dtype=torch.float64, device="cuda")
    d.backward_fp64(w.data_ptr(), g.data_ptr())
    torch.cuda.synchronize()
    return g.cpu().numpy()


def test_fp64_adjoint_of_fp32_records_matches_central_differences(cuda):
    """kt_diff_backward_fp64 on an FP32 object differentiates its records replayed in double
    (the model of kt_diff_replay_fp64), segment starts included: the loss gradient matches that
    model's central differences to 1e-4 in all four parameters, r_out included, where the FP32
    adjoint carries the float rounding of its hit states."""
    _, _, d = make(kt.PREC_FP32)
    hdr = forward(cuda, d, THETA)
    fd, mask = central_differences(cuda, d, replay_fp64)
    lit = hdr[:, :3].sum(1) > 0
    assert int(mask.sum()) <= 0.02 * int(lit.sum())
    n = SIZE * SIZE
    rng = np.random.default_rng(1)
    w = cuda.tensor((rng.standard_normal((n, 4)) + 1.0).astype(np.float32), device="cuda")
    w[:, 3] = 0
    w[mask] = 0
    g64 = backward_fp64(cuda, d, w)
    g32 = backward(cuda, d, w)
    for j in range(4):
        ref = float((fd[j] * w[:, :3].double()).sum())
        print(NAMES[j], g64[j], g32[j], ref, abs(g64[j] - ref) / abs(ref))
        assert abs(g64[j] - ref) <= 1e-4 * abs(ref), (NAMES[j], g64[j], ref)
    # and the FP32 adjoint of the same records is close to it where it is accurate
    for j in range(3):
        assert abs(g32[j] - g64[j]) <= 1e-3 * abs(g64[j]), NAMES[j]
    d.close()


def test_fp32_adjoint_tracks_fp64(cuda):
    n = SIZE * SIZE
    rng = np.random.default_rng(4)
    w = cuda.tensor((rng.standard_normal((n, 4)) + 1.0).astype(np.float32), device="cuda")
    w[:, 3] = 0
    g = {}
    for prec in (kt.PREC_FP64, kt.PREC_FP32):
        _, _, d = make(prec)
        forward(cuda, d, THETA)
        g[prec] = backward(cuda, d, w)
        d.close()
    for j in range(3):
        assert abs(g[kt.PREC_FP32][j] - g[kt.PREC_FP64][j]) <= 2e-3 * abs(g[kt.PREC_FP64][j]), NAMES[j]
    assert abs(g[kt.PREC_FP32][3] - g[kt.PREC_FP64][3]) <= 5e-2 * abs(g[kt.PREC_FP64][3])


def test_fp64_adjoint_matches_oracle_reference_gradient(cuda):
    """The FP64 adjoint against the f64 CPU reference gradient (the oracle's forward-mode
    restatement of the same frozen-step trace), on the pixels whose images agree to 1e-6 (the
    others took a different step sequence)."""
    import oracle
    size = 48
    n = size * size
    cfg, view = workloads.c5(size, kt.PREC_FP64)
    d = kt.Diff(cfg, view)
    hdr = cuda.zeros((n, 4), device="cuda")
    err = cuda.zeros(2, dtype=cuda.int32, device="cuda")
    d.forward(THETA, hdr.data_ptr(), err.data_ptr())
    cuda.cuda.synchronize()
    col, dcol, _ = oracle.diff_render(cfg, view, THETA)
    img = hdr[:, :3].double().cpu().numpy()
    same = np.abs(img - col).max(1) <= 1e-6 * (np.abs(col).max(1) + 1e-12)
    assert same.mean() > 0.95
    rng = np.random.default_rng(1)
    w = rng.standard_normal((n, 3)) + 1.0
    w[~same] = 0.0
    W = cuda.zeros((n, 4), device="cuda")
    W[:, :3] = cuda.tensor(w, dtype=cuda.float32, device="cuda")
    g = backward(cuda, d, W)
    ref = np.einsum("pc,pcj->j", W[:, :3].double().cpu().numpy(), dcol)
    for j, tol in enumerate((1e-5, 1e-5, 1e-6, 1e-4)):
        assert abs(g[j] - ref[j]) <= tol * abs(ref[j]), (NAMES[j], g[j], ref[j])
    d.close()


@pytest.mark.parametrize("size", [(1, 1), (17, 15), (33, 48), (70, 5)])
def test_diff_ragged_frames(cuda, size):
    """Frames that are not whole 16x16 tiles: the recorded forward is the stated-physics trace bit for
    bit on every pixel, and the FP32 loss gradient agrees with the FP64 one to the two models'
    distance (their step sequences differ at the tolerance: 1e-2 of the gradient's norm)."""
    import torch
    grads = {}
    for prec in (kt.PREC_FP32, kt.PREC_FP64):
        cfg, view = workloads.c5(64, prec)
        cfg.width, cfg.height = size
        n = size[0] * size[1]
        d = kt.Diff(cfg, view)
        hdr = torch.full((n, 4), float("nan"), device="cuda")
        err = torch.zeros(2, dtype=torch.int32, device="cuda")
        g = torch.zeros(4, dtype=torch.float64, device="cuda")
        d.forward(workloads.C5_START, hdr.data_ptr(), err.data_ptr())
        w = torch.ones((n, 4), device="cuda")
        d.backward(w.data_ptr(), g.data_ptr())
        torch.cuda.synchronize()
        assert bool((hdr[:, 3] == 1.0).all()) and bool(torch.isfinite(hdr).all())
        grads[prec] = g.cpu().numpy()
        if prec == kt.PREC_FP32:
            c = cfg.copy()
            th = workloads.C5_START
            c.spin, c.disk_outer_radius = th[0], th[3]
            c.disk_temperature_scale = float(np.float32(view.base_temperature_scale * th[2]))
            cam, _ = kt.diff_orbit_camera(view.observer_r, th[1], view.azimuth_deg, view.fov_deg)
            bb = kt.generate_blackbody_lut(c.lut_size, c.lut_max_temp, c.wavelength_start, c.wavelength_end,
                                           c.wavelength_step)
            ctx = kt.Context(c, luts=(bb, kt.generate_disk_lut(kt.build_kerr_params(c), c.disk_outer_radius, c.lut_size)))
            ref = torch.zeros((n, 4), device="cuda")
            ctx.trace(cam, ref.data_ptr(), err.data_ptr(), 0, kt.SCHED_PLAIN)
            torch.cuda.synchronize()
            assert torch.equal(hdr, ref)
            ctx.close()
        d.close()
    a, b = grads[kt.PREC_FP32], grads[kt.PREC_FP64]
    assert np.linalg.norm(a - b) <= 1e-2 * np.linalg.norm(b) + 1e-12
