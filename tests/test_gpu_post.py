"""Post-processing on the GPU: the product's bloom / post / fused kernels against the reference's
bloom_horizontal + post_process (oracle/_ref) on identical HDR input — bit-identical bloom
buffers and 0x00RRGGBB images — and against the oracle's double-precision post (±1 per byte)."""
from __future__ import annotations

import numpy as np
import pytest

import kerrtrace_b200 as kt
from kerrtrace_b200 import workloads

pytestmark = pytest.mark.gpu


def _bloom_consts(cfg):
    radius = int(np.ceil(np.float32(cfg.bloom_radius))) if cfg.bloom_radius > 0 else 0
    sigma = float(np.float32(np.float32(cfg.bloom_radius) / np.float32(3.0)))
    active = int(bool(cfg.bloom_enabled) and radius > 0 and cfg.bloom_intensity > 0)
    return radius, sigma, active


def _hdr_input(torch, cfg, seed):
    """Synthetic HDR with a wide dynamic range, exact zeros, NaN-free."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    n = cfg.width * cfg.height
    base = torch.rand((n, 4), generator=g) ** 6 * 20.0
    base[torch.rand(n, generator=g) < 0.2] = 0.0
    base[:, 3] = 1.0
    return base.cuda()


@pytest.mark.parametrize("name,size,radius", [("t1", None, None), ("t2", None, None), ("c2", (333, 190), None),
                                              ("c2", (64, 40), 48.0), ("t1", (50, 70), 0.0),
                                              ("c2", (96, 300), 70.0), ("c2", (72, 260), 95.0),
                                              ("c2", (80, 90), 100.0), ("t1", (1, 1), None),
                                              ("c2", (1920, 1080), None)])
def test_post_bit_identical_to_reference(cuda, orc, name, size, radius):
    cfg, _ = workloads.scene(name)
    if size:
        cfg = workloads.scaled(cfg, *size)
    if radius is not None:
        cfg.bloom_radius = radius
    R, sigma, active = _bloom_consts(cfg)
    hdr = _hdr_input(cuda, cfg, 7)
    n = cfg.width * cfg.height
    ctx = kt.Context(cfg)
    ref = orc.RefKernel(name)
    bloom_o = cuda.zeros((n, 4), device="cuda")
    bloom_r = cuda.zeros((n, 4), device="cuda")
    img_o = cuda.zeros(n, dtype=cuda.int32, device="cuda")
    img_f = cuda.zeros(n, dtype=cuda.int32, device="cuda")
    img_r = cuda.zeros(n, dtype=cuda.int32, device="cuda")
    if active:
        ctx.bloom_horizontal(hdr.data_ptr(), bloom_o.data_ptr())
        ref.bloom(hdr.data_ptr(), bloom_r.data_ptr(), cfg, R, sigma, active)
    ctx.post_process(hdr.data_ptr(), bloom_o.data_ptr(), img_o.data_ptr())
    ctx.post_fused(hdr.data_ptr(), img_f.data_ptr())
    ref.post(hdr.data_ptr(), bloom_r.data_ptr(), img_r.data_ptr(), cfg, R, sigma, cfg.bloom_intensity, active)
    cuda.cuda.synchronize()
    bo, br = bloom_o.cpu().numpy(), bloom_r.cpu().numpy()
    io, i_f, ir = (t.cpu().numpy().view(np.uint32) for t in (img_o, img_f, img_r))
    if active:
        assert np.array_equal(bo.view(np.uint32), br.view(np.uint32))
    assert np.array_equal(io, ir)
    assert np.array_equal(i_f, ir)
    assert np.all(ir >> 24 == 0)
    # oracle (double precision) agrees within one code value per channel
    exp = orc.post(hdr.cpu().numpy(), cfg.width, cfg.height, R if active else 0, sigma, cfg.bloom_intensity)
    d = np.max(np.abs(np.stack([(ir >> s) & 255 for s in (16, 8, 0)]).astype(int) -
                      np.stack([(exp >> s) & 255 for s in (16, 8, 0)]).astype(int)), axis=0)
    assert d.max() <= 1, np.bincount(d)
    ctx.close()
    ref.close()


def test_post_rejects_misaligned_buffers(cuda):
    """The post entry points read and write float4 pixels: a pointer off the 16-byte grid (or an
    image pointer off the 4-byte grid) is refused on the host, before any launch."""
    cfg, _ = workloads.scene("t1")
    n = cfg.width * cfg.height
    ctx = kt.Context(cfg)
    hdr = cuda.zeros((n + 1, 4), device="cuda")
    bloom = cuda.zeros((n + 1, 4), device="cuda")
    img = cuda.zeros(n + 1, dtype=cuda.int32, device="cuda")
    calls = [lambda: ctx.post_fused(hdr.data_ptr() + 4, img.data_ptr()),
             lambda: ctx.post_fused(hdr.data_ptr(), img.data_ptr() + 2),
             lambda: ctx.bloom_horizontal(hdr.data_ptr() + 8, bloom.data_ptr()),
             lambda: ctx.bloom_horizontal(hdr.data_ptr(), bloom.data_ptr() + 4),
             lambda: ctx.post_process(hdr.data_ptr(), bloom.data_ptr() + 12, img.data_ptr())]
    for call in calls:
        with pytest.raises(kt.KtError) as e:
            call()
        assert e.value.status == kt.KT_ERR_INVALID_ARG and "aligned" in str(e.value)
    ctx.post_fused(hdr.data_ptr(), img.data_ptr())  # aligned: runs
    cuda.cuda.synchronize()
    ctx.close()


@pytest.mark.parametrize("size,radius", [(None, None), ((333, 190), 24.0), ((64, 40), 48.0), ((1, 1), None)])
def test_stated_physics_bloom_threshold(cuda, orc, size, radius):
    """Stated physics blooms only the luminance above the threshold (the source of each in-image
    value is scaled in place after staging).  The fused pair (column-major bloom buffer) equals
    the separate passes bit for bit, and both agree with the oracle's double-precision post to
    one code value per channel."""
    cfg, _ = workloads.scene("c2")
    cfg = workloads.scaled(cfg, *(size or (160, 96)))
    cfg.mode = 1
    cfg.bloom_threshold = 1.0
    if radius is not None:
        cfg.bloom_radius = radius
    R, sigma, active = _bloom_consts(cfg)
    assert active
    hdr = _hdr_input(cuda, cfg, 11)
    n = cfg.width * cfg.height
    ctx = kt.Context(cfg)
    bloom = cuda.zeros((n, 4), device="cuda")
    img_s = cuda.zeros(n, dtype=cuda.int32, device="cuda")
    img_f = cuda.zeros(n, dtype=cuda.int32, device="cuda")
    ctx.bloom_horizontal(hdr.data_ptr(), bloom.data_ptr())
    ctx.post_process(hdr.data_ptr(), bloom.data_ptr(), img_s.data_ptr())
    ctx.post_fused(hdr.data_ptr(), img_f.data_ptr())
    cuda.cuda.synchronize()
    i_s, i_f = (t.cpu().numpy().view(np.uint32) for t in (img_s, img_f))
    assert np.array_equal(i_s, i_f)
    exp = orc.post(hdr.cpu().numpy(), cfg.width, cfg.height, R, sigma, cfg.bloom_intensity, 1, cfg.bloom_threshold)
    d = np.max(np.abs(np.stack([(i_f >> s) & 255 for s in (16, 8, 0)]).astype(int) -
                      np.stack([(exp >> s) & 255 for s in (16, 8, 0)]).astype(int)), axis=0)
    assert d.max() <= 1, np.bincount(d)
    # the threshold matters: the reference semantics' bloom of the same input differs
    cfg0 = cfg.copy()
    cfg0.mode = 0
    ctx0 = kt.Context(cfg0)
    img_0 = cuda.zeros(n, dtype=cuda.int32, device="cuda")
    ctx0.post_fused(hdr.data_ptr(), img_0.data_ptr())
    cuda.cuda.synchronize()
    if n > 1:
        assert not np.array_equal(img_0.cpu().numpy().view(np.uint32), i_f)
    ctx0.close()
    ctx.close()


@pytest.mark.parametrize("size,radius", [((1, 1), 24.0), ((7, 3), 1.0), ((33, 65), 2.0), ((65, 129), 3.5), ((64, 64), 4.0),
                                         ((63, 127), 24.0), ((1, 200), 24.0), ((200, 1), 24.0), ((641, 97), 90.0),
                                         ((400, 60), 163.0), ((50, 40), 300.0)])
def test_post_tiles_against_oracle(cuda, orc, size, radius):
    """Tiles of line pairs at their edges (odd lines and positions, frames smaller than a tile, radii
    with fewer taps than a thread's outputs and up to the largest that fits): the fused pair equals
    the separate passes bit for bit, the bloom buffer is the double-precision horizontal Gaussian to
    float rounding (sum of 2R + 1 products: relative error (2R + 2) 2^-24, plus the fast exponential's
    2e-6 per weight), and the image is the oracle's to one code value.  Radius 300 is beyond the
    tiles: only the vertical pass takes it (bloom buffer given)."""
    cfg, _ = workloads.scene("t1")
    cfg = workloads.scaled(cfg, *size)
    cfg.bloom_radius = radius
    R, sigma, active = _bloom_consts(cfg)
    w, h = size
    hdr = _hdr_input(cuda, cfg, 5)
    ctx = kt.Context(cfg)
    bloom = cuda.zeros((w * h, 4), device="cuda")
    img_s, img_f = (cuda.zeros(w * h, dtype=cuda.int32, device="cuda") for _ in range(2))
    src = hdr.cpu().numpy().astype(np.float64).reshape(h, w, 4)[..., :3]
    k = np.exp(-np.arange(-R, R + 1) ** 2 / (2 * sigma ** 2))
    full = np.zeros((h, w + 2 * R, 3))
    full[:, R:R + w] = src
    ones = np.zeros(w + 2 * R)
    ones[R:R + w] = 1.0
    exp_b = sum(k[i] * full[:, i:i + w] for i in range(2 * R + 1)) / sum(k[i] * ones[i:i + w] for i in range(2 * R + 1))[None, :, None]
    if radius <= 163:
        ctx.bloom_horizontal(hdr.data_ptr(), bloom.data_ptr())
        ctx.post_fused(hdr.data_ptr(), img_f.data_ptr())
    else:
        with pytest.raises(kt.KtError):
            ctx.bloom_horizontal(hdr.data_ptr(), bloom.data_ptr())
        bloom[:, :3] = cuda.from_numpy(exp_b.reshape(-1, 3).astype(np.float32)).cuda()
    ctx.post_process(hdr.data_ptr(), bloom.data_ptr(), img_s.data_ptr())
    cuda.cuda.synchronize()
    got = bloom.cpu().numpy().reshape(h, w, 4)[..., :3].astype(np.float64)
    assert np.max(np.abs(got - exp_b) / np.maximum(np.abs(exp_b), 1e-30)) < (2 * R + 2) * 2.0 ** -24 + 4e-6
    i_s = img_s.cpu().numpy().view(np.uint32)
    if radius <= 163:
        assert np.array_equal(i_s, img_f.cpu().numpy().view(np.uint32))
    exp = orc.post(hdr.cpu().numpy(), w, h, R, sigma, cfg.bloom_intensity)
    d = np.max(np.abs(np.stack([(i_s >> s) & 255 for s in (16, 8, 0)]).astype(int) -
                      np.stack([(exp >> s) & 255 for s in (16, 8, 0)]).astype(int)), axis=0)
    assert d.max() <= 1, np.bincount(d)
    ctx.close()


@pytest.mark.parametrize("size,radius", [((33, 17), 2.0), ((333, 217), 24.0), ((960, 540), 24.0)])
@pytest.mark.parametrize("graph", [False, True])
def test_overlapped_launches_keep_stream_order(cuda, size, radius, graph):
    """Post passes issued one behind the other on two streams, each behind a kernel or a copy that
    rewrites its input (directly and as one captured graph), equal the passes run one at a time."""
    cfg, _ = workloads.scene("t1")
    cfg = workloads.scaled(cfg, *size)
    cfg.bloom_radius = radius
    n = size[0] * size[1]
    inputs = [_hdr_input(cuda, cfg, 11 + i) for i in range(3)]
    ctx = [kt.Context(cfg) for _ in range(2)]
    hdr = [cuda.zeros((n, 4), device="cuda") for _ in ctx]
    img = [cuda.zeros(n, dtype=cuda.int32, device="cuda") for _ in ctx]
    want = []
    for x in inputs:
        ctx[0].post_fused(x.data_ptr(), img[0].data_ptr())
        cuda.cuda.synchronize()
        want.append(img[0].clone())
    got = [[cuda.zeros_like(i) for _ in range(12)] for i in img]

    def issue(q, stream):
        for it in range(12):
            x = inputs[(it + q) % 3]
            (cuda.mul(x, 1.0, out=hdr[q]) if it % 2 else hdr[q].copy_(x))
            ctx[q].post_fused(hdr[q].data_ptr(), img[q].data_ptr(), stream.cuda_stream)
            got[q][it].copy_(img[q])

    streams = [cuda.cuda.Stream() for _ in ctx]
    graphs = []
    cuda.cuda.synchronize()
    for q, st in enumerate(streams):
        if graph:
            g = cuda.cuda.CUDAGraph()
            with cuda.cuda.graph(g, stream=st):
                issue(q, st)
            graphs.append(g)
        else:
            with cuda.cuda.stream(st):
                issue(q, st)
    for g in graphs:
        g.replay()
    cuda.cuda.synchronize()
    for q in range(2):
        for it in range(12):
            assert cuda.equal(got[q][it], want[(it + q) % 3]), (q, it)


def test_post_passes_of_two_radii_from_two_threads(cuda):
    """Two host threads whose contexts need different amounts of shared memory (radii 90 and 60, both
    above the default limit) issue their passes at the same time: every call succeeds, and the images
    are those of calls made one after the other."""
    import threading
    ctx, hdr, img, want, failed = [], [], [], [], []
    for i, radius in enumerate((90.0, 60.0)):
        cfg, _ = workloads.scene("t1")
        cfg = workloads.scaled(cfg, 64, 40)
        cfg.bloom_radius = radius
        ctx.append(kt.Context(cfg))
        hdr.append(_hdr_input(cuda, cfg, 21 + i))
        img.append(cuda.zeros(64 * 40, dtype=cuda.int32, device="cuda"))
        ctx[i].post_fused(hdr[i].data_ptr(), img[i].data_ptr())
        cuda.cuda.synchronize()
        want.append(img[i].clone())
    streams = [cuda.cuda.Stream() for _ in ctx]
    start = threading.Barrier(2)

    def issue(i):
        start.wait()
        for _ in range(4000):
            try:
                ctx[i].post_fused(hdr[i].data_ptr(), img[i].data_ptr(), streams[i].cuda_stream)
            except kt.KtError as e:
                failed.append(str(e))

    threads = [threading.Thread(target=issue, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    cuda.cuda.synchronize()
    assert not failed, (len(failed), failed[0])
    for i in range(2):
        assert cuda.equal(img[i], want[i])


@pytest.mark.parametrize("radius,taken", [(165.0, True), (165.5, False), (229.0, False), (230.0, False)])
def test_largest_radius_of_each_pass(cuda, orc, radius, taken):
    """The horizontal and the fused pass take radii up to 165; the vertical pass takes all of these, tiled
    up to 229 and one pixel per thread beyond: the image is the oracle's to one code value."""
    cfg, _ = workloads.scene("t1")
    cfg = workloads.scaled(cfg, 40, 90)
    cfg.bloom_radius = radius
    R, sigma, _ = _bloom_consts(cfg)
    w, h = cfg.width, cfg.height
    hdr = _hdr_input(cuda, cfg, 31)
    ctx = kt.Context(cfg)
    bloom = cuda.zeros((w * h, 4), device="cuda")
    img_s, img_f = (cuda.zeros(w * h, dtype=cuda.int32, device="cuda") for _ in range(2))
    if taken:
        ctx.bloom_horizontal(hdr.data_ptr(), bloom.data_ptr())
        ctx.post_fused(hdr.data_ptr(), img_f.data_ptr())
    else:
        for refused in (lambda: ctx.bloom_horizontal(hdr.data_ptr(), bloom.data_ptr()),
                        lambda: ctx.post_fused(hdr.data_ptr(), img_f.data_ptr())):
            with pytest.raises(kt.KtError):
                refused()
        k = np.exp(-np.arange(-R, R + 1) ** 2 / (2 * sigma ** 2))
        src = np.zeros((h, w + 2 * R, 4))
        src[:, R:R + w, :3] = hdr.cpu().numpy().reshape(h, w, 4)[..., :3]
        src[:, R:R + w, 3] = 1.0
        b = sum(k[i] * src[:, i:i + w] for i in range(2 * R + 1))
        bloom[:, :3] = cuda.from_numpy((b[..., :3] / b[..., 3:]).reshape(-1, 3).astype(np.float32)).cuda()
    ctx.post_process(hdr.data_ptr(), bloom.data_ptr(), img_s.data_ptr())
    cuda.cuda.synchronize()
    got = img_s.cpu().numpy().view(np.uint32)
    if taken:
        assert np.array_equal(got, img_f.cpu().numpy().view(np.uint32))
    exp = orc.post(hdr.cpu().numpy(), w, h, R, sigma, cfg.bloom_intensity)
    d = np.max(np.abs(np.stack([(got >> s) & 255 for s in (16, 8, 0)]).astype(int) -
                      np.stack([(exp >> s) & 255 for s in (16, 8, 0)]).astype(int)), axis=0)
    assert d.max() <= 1, np.bincount(d)
    ctx.close()
