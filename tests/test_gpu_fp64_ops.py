"""The FP64 path's reciprocal, division and square root (Goldschmidt's iterations with Markstein's last
step) against CUDA's own operators and sqrt(), bit for bit: random operands over the range, results
next to the midpoint of two doubles, and the ends of the range."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

INV, DIV, SQRT = 0, 1, 2
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def probe():
    import oracle.build as obuild
    L = C.CDLL(str(obuild.PROBE_LIB))
    L.ktp_fp64_op.argtypes = [C.c_int, C.c_longlong] + 4 * [C.c_void_p]
    L.ktp_fp64_attempt.argtypes = 2 * [C.c_double] + 3 * [C.c_void_p]
    L.ktp_fp64_random.argtypes = [C.c_int, C.c_ulonglong, C.c_int, C.c_int, C.c_int, C.c_void_p]
    return L


def run(cuda, probe, op, a, b=None):
    n = len(a)
    d = [cuda.tensor(np.asarray(v, np.float64), device="cuda") for v in (a, a if b is None else b)]
    out = [cuda.zeros(n, dtype=cuda.float64, device="cuda") for _ in range(2)]
    cuda.cuda.synchronize()
    assert probe.ktp_fp64_op(op, n, *[C.c_void_p(t.data_ptr()) for t in (*d, *out)]) == 0
    return [t.cpu().numpy() for t in out]


def same(a, b):
    return (a.view(np.uint64) == b.view(np.uint64)) | (np.isnan(a) & np.isnan(b))


@pytest.mark.parametrize("op,exponent", [(INV, 30), (INV, 1000), (DIV, 30), (DIV, 450), (SQRT, 30), (SQRT, 900)])
def test_random_operands(cuda, probe, op, exponent):
    """2^28 operands each; exponents up to those whose quotients and remainders stay normal."""
    bad = cuda.zeros(1, dtype=cuda.int64, device="cuda")
    cuda.cuda.synchronize()
    assert probe.ktp_fp64_random(op, 0x9e3779b97f4a7c15 + 2 * exponent, 8192, 256, exponent, C.c_void_p(bad.data_ptr())) == 0
    assert int(bad) == 0


def near_midpoint_divisors():
    """b = 2^53 - j with j odd: b (2^53 + j) = 2^106 - j^2, so 1/b lies j^2 2^-106 (relative) above the
    midpoint (2^53 + j) 2^-106 of two doubles, as close as a reciprocal gets."""
    return [float(2 ** 53 - j) for j in range(3, 40001, 2)]


def near_midpoint_quotients(rng, count):
    """a 2^54 = s mod b with a small s: a / b lies s / (b 2^54) from (a 2^54 - s) / b 2^-54, a midpoint
    when that integer is odd."""
    a, b = [], []
    while len(a) < count:
        d = int(rng.integers(2 ** 52, 2 ** 53)) | 1
        s = int(rng.integers(1, 64)) * (1 if rng.integers(2) else -1)
        n = s * pow(2, -54, d) % d
        if 2 * n > d and ((n << 54) - s) // d % 2 == 1:
            a.append(float(n))
            b.append(float(d))
    return a, b


def near_midpoint_squares(count):
    """M odd of 54 bits with M^2 = c mod 2^k, c small: sqrt((M^2 - c) / 2^k) lies next to M 2^(-k/2), a
    midpoint.  c = 1 mod 8 has four square roots modulo 2^k."""
    out = []
    for k in (54, 55):
        for c in range(1 - 8 * count, 1 + 8 * count, 8):
            m = 1
            for i in range(3, k):
                if (m * m - c) % 2 ** (i + 1):
                    m += 2 ** (i - 1)
            for r in {m % 2 ** k, -m % 2 ** k, (m + 2 ** (k - 1)) % 2 ** k, (2 ** (k - 1) - m) % 2 ** k}:
                x = (r * r - c) >> k
                if 2 ** 53 <= r and r < 2 ** 54 and (r * r - c) % 2 ** k == 0 and 2 ** 52 <= x < 2 ** 53:
                    out.append(float(x) * (2.0 if k % 2 else 1.0))
    return out


def test_results_next_to_a_midpoint(cuda, probe):
    got, want = run(cuda, probe, INV, near_midpoint_divisors())
    assert same(got, want).all(), int((~same(got, want)).sum())
    got, want = run(cuda, probe, DIV, *near_midpoint_quotients(np.random.default_rng(3), 20000))
    assert same(got, want).all(), int((~same(got, want)).sum())
    x = near_midpoint_squares(4000)
    assert len(x) > 8000
    got, want = run(cuda, probe, SQRT, x)
    assert same(got, want).all(), int((~same(got, want)).sum())
    # the one divisor that the last step does not cover, a significand of all ones: a neighbour at most
    got, want = run(cuda, probe, INV, [2.0 - 2.0 ** -52, 2.0 ** 53 - 1, 1.0 - 2.0 ** -53])
    assert (np.abs(got.view(np.int64) - want.view(np.int64)) <= 1).all()


def test_ends_of_the_range(cuda, probe):
    """What the comment of the functions promises beside the normal range."""
    inf, nan, tiny, big = np.inf, np.nan, 2.0 ** -1074, 2.0 ** 1023
    got, want = run(cuda, probe, SQRT, [0.0, -0.0, inf, nan, -1.0, -inf, 2.0 ** -1022, np.finfo(np.float64).max])
    assert same(got, want).all(), (got, want)
    got, want = run(cuda, probe, INV, [-3.0, 2.0 ** -1022, 2.0 ** 1021, -2.0 ** -1000, 1.0])
    assert same(got, want).all(), (got, want)
    got, _ = run(cuda, probe, INV, [0.0, tiny, inf, nan])
    assert np.isnan(got).all(), got
    got, want = run(cuda, probe, DIV, [0.0, 0.0, 1.0], [3.0, big / 4, 1.0])
    assert same(got, want).all(), (got, want)
    # never finite where the operator gives NaN or an infinity
    a = [inf, inf, nan, 1.0, 1.0, 1.0, 0.0, big, 1e200, 1.0]
    b = [1.0, inf, 1.0, nan, 0.0, tiny, 0.0, 2.0 ** -1000, 1e-200, inf]
    got, want = run(cuda, probe, DIV, a, b)
    assert np.isnan(got).all(), (got, want)


@pytest.mark.parametrize("component", [0, 1, 2])
@pytest.mark.parametrize("h,accepted", [(1e-3, True), (1e14, False)])
def test_a_step_with_one_error_component_out_of_range_is_rejected(cuda, probe, component, h, accepted):
    """Straight motion along one axis (no mass), whose k1 is not its velocity: that component's error is
    h x 71/57600, the other five are exactly 0.  Over scales of 5e-300 and more the quotient is 6e309
    to 2.4e310 for h = 1e14, beyond the doubles: an infinite error, and a step that has to be tried
    again.  The accepted step has h = 1e-3 and scales of 5 and more."""
    x = np.zeros(15)
    x[:3] = 20.0, 5.0, 7.0
    x[3 + component] = 1.0
    x[6 + component] = 2.0
    x[12], x[13], x[14] = -1.0, h, 1.0 if accepted else 1e-300
    d_in = cuda.tensor(x, device="cuda")
    out = cuda.zeros(8, dtype=cuda.float64, device="cuda")
    err = cuda.zeros(2, dtype=cuda.int32, device="cuda")
    cuda.cuda.synchronize()
    assert probe.ktp_fp64_attempt(0.0, 0.0, *[C.c_void_p(t.data_ptr()) for t in (d_in, out, err)]) == 0
    got = out.cpu().numpy()
    if accepted:
        assert got[7] == 0 and got[component] != x[component]
    else:
        assert got[7] == 1 and np.array_equal(got[:6], x[:6]) and got[6] == 0.0
