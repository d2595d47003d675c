"""The orders in which the persistent trace, the batch, the views call and the recording forward take
the pixels of a frame (host code, no device): every pixel once, and few idle lanes in a launch that
fills the GPU."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

WARPS = 148 * 16


@pytest.fixture(scope="module")
def probe():
    import oracle.build as obuild
    L = C.CDLL(str(obuild.PROBE_LIB))
    L.ktp_frame_pixels.argtypes = [C.c_int, C.c_int, C.c_int, C.c_longlong, C.c_void_p]
    L.ktp_unit_count.argtypes = 4 * [C.c_int]
    L.ktp_unit_count.restype = C.c_uint
    L.ktp_take_strips.argtypes = [C.c_int, C.c_int, C.c_uint, C.c_uint]
    return L


def pixels(probe, w, h, strips, n):
    out = np.zeros(n, np.int32)
    probe.ktp_frame_pixels(w, h, strips, n, out.ctypes.data)
    return out


@pytest.mark.parametrize("w", [1, 2, 3, 4, 5, 7, 8, 9, 11, 12, 13, 16, 17, 20, 25, 31, 33, 64, 100, 111, 129])
@pytest.mark.parametrize("strips", [0, 1])
def test_every_pixel_once(probe, w, strips):
    for h in [*range(1, 22), 31, 33, 48, 49, 64, 65, 130]:
        units = probe.ktp_unit_count(w, h, 1, strips)
        p = pixels(probe, w, h, strips, 32 * units + 70)
        inside = p[p >= 0]
        assert len(inside) == w * h and np.array_equal(np.sort(inside), np.arange(w * h)), (w, h)
        assert (p[32 * units:] == -1).all()
        last = np.flatnonzero(p >= 0)[-1]
        for S in (1, 2, 3, 5, 8, 10, 16, 31, 32):  # the units reach the last pixel
            assert last < probe.ktp_unit_count(w, h, S, strips) * (32 // S), (w, h, S)


@pytest.mark.parametrize("w,h", [(32768, 1), (1, 32768), (32768, 3), (5, 32768), (32768, 7), (9, 32768), (17, 32768),
                                 (8000, 17), (33, 4001), (100, 2000), (1920, 1080), (960, 540), (640, 640)])
def test_large_launches_have_few_idle_lanes(probe, w, h):
    """In the order that a launch of more patches than warps takes, 15 of 16 lanes of the units with a
    pixel have one, and a run of 32 lies within 32 columns and 32 rows, unless it passes from the
    foot of one strip of columns to the head of the next."""
    patches = probe.ktp_unit_count(w, h, 1, 0)
    strips = probe.ktp_take_strips(w, h, patches, WARPS)
    assert patches > WARPS and probe.ktp_take_strips(w, h, patches, patches) == 0
    p = pixels(probe, w, h, strips, 32 * probe.ktp_unit_count(w, h, 1, strips)).reshape(-1, 32)
    used = int((p >= 0).any(1).sum())
    assert 16 * w * h >= 15 * 32 * used, (used, w * h / 32)
    run = p[(p >= 0).all(1)]
    wide = (np.ptp(run % w, axis=1) > 32) | (np.ptp(run // w, axis=1) > 32)
    assert wide.sum() <= w // 6 + 1
