// device_probe.cu — runs single device functions of the product on given operands.  TEST
// INFRASTRUCTURE ONLY: built from the product's headers with the flags of its kernels, so that
// functions which no entry point exposes by themselves can be compared with CUDA's own.
//
// Every launch is one thread per operand, in bounds by construction; the C functions with launches
// take device pointers, run on the legacy stream and return the CUDA status after a
// synchronisation.  The unit order is host code and needs no device.
#include <cuda_runtime.h>
#include <stdint.h>

#include "kt_internal.h"
#include "kt_ray.cuh"

namespace {

// op 0: 1 / a, 1: a / b, 2: sqrt(a); ours into `got`, the operators and sqrt() into `want`.
__global__ void fp64_op_kernel(int op, long long n, const double* a, const double* b, double* got, double* want) {
    using O = ktd::Ops<double>;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x = a[i];
    if (op == 0) {
        got[i] = O::inv(x);
        want[i] = 1.0 / x;
    } else if (op == 1) {
        got[i] = O::ratio(x, b[i]);
        want[i] = x / b[i];
    } else {
        got[i] = O::sqrt_rn(x);
        want[i] = sqrt(x);
    }
}

// Mix of a 64-bit counter (a bijection, so operands do not repeat).
__device__ __forceinline__ uint64_t mix(uint64_t x) {
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}
// A positive double with a random significand and a binary exponent in [-e, e].
__device__ __forceinline__ double operand(uint64_t r, int e) {
    const uint64_t m = mix(r);
    const int ex = (int)(mix(~r) % (uint64_t)(2 * e + 1)) - e;
    return __longlong_as_double((long long)((m >> 12) | (uint64_t)(1023 + ex) << 52));
}

// Counts the random operands (exponents in [-e, e]) whose result differs from the operators'.
__global__ void fp64_random_kernel(int op, uint64_t first, uint64_t per_thread, int e, unsigned long long* differing) {
    using O = ktd::Ops<double>;
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned bad = 0;
    for (uint64_t k = 0; k < per_thread; ++k) {
        const uint64_t r = first + 2 * (t * per_thread + k);
        const double x = operand(r, e), y = operand(r + 1, e);
        const double got = op == 0 ? O::inv(x) : op == 1 ? O::ratio(x, y) : O::sqrt_rn(x);
        const double want = op == 0 ? 1.0 / x : op == 1 ? x / y : sqrt(x);
        bad += __double_as_longlong(got) != __double_as_longlong(want) ? 1u : 0u;
    }
    if (bad) atomicAdd(differing, (unsigned long long)bad);
}

// One FP64 attempt of the stated physics from the state in[0..5] with k1 in[6..11], p_t, step size and
// tolerance in[12..14]; out: the state after it, the next step size, the attempts spent on the
// step (0 after a commit).
__global__ void fp64_attempt_kernel(const __grid_constant__ ktd::Scene sc, const double* in, double* out,
                                    uint32_t* err) {
    ktd::RayRun<double> ry;
    ktd::Tally tl;
    tl.clear();
    for (int c = 0; c < 6; ++c) {
        ry.s[c] = in[c];
        ry.k1[c] = in[6 + c];
    }
    ry.pt = in[12];
    ry.kt = 0.0;
    ry.h = in[13];
    ry.tol = in[14];
    ry.col[0] = ry.col[1] = ry.col[2] = 0.0;
    ry.tau = 1.0;
    ry.step = ry.attempt = 0;
    ktd::ray_advance<double, 1, false, false>(ry, sc, err, tl, ktd::kRayGoing);
    for (int c = 0; c < 6; ++c) out[c] = ry.s[c];
    out[6] = ry.h;
    out[7] = ry.attempt;
}

}  // namespace

extern "C" {

// mass, spin: of the hole; the disk, the sky and the escape radius are out of reach.
int ktp_fp64_attempt(double mass, double spin, const double* in, double* out, uint32_t* err) {
    ktd::Scene sc = {};
    sc.M_d = mass;
    sc.a_d = spin;
    sc.aa_d = spin * spin;
    sc.M = (float)mass;
    sc.max_steps = sc.max_attempts = 10;
    sc.escape_d = 1e300;
    sc.disk_inner_d = 1e299;
    sc.disk_outer_d = 1e300;
    sc.base_tol_d = 1e-6;
    sc.mode = 1;
    sc.precision = 2;
    fp64_attempt_kernel<<<1, 1>>>(sc, in, out, err);
    const cudaError_t e = cudaGetLastError();
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}

int ktp_fp64_op(int op, long long n, const double* a, const double* b, double* got, double* want) {
    if (n <= 0 || op < 0 || op > 2) return (int)cudaErrorInvalidValue;
    fp64_op_kernel<<<(unsigned)((n + 127) / 128), 128>>>(op, n, a, b, got, want);
    const cudaError_t e = cudaGetLastError();
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}

int ktp_fp64_random(int op, unsigned long long first, int blocks, int per_thread, int max_exponent,
                    unsigned long long* differing) {
    if (blocks <= 0 || per_thread <= 0 || op < 0 || op > 2 || max_exponent < 0 || max_exponent > 1000)
        return (int)cudaErrorInvalidValue;
    fp64_random_kernel<<<blocks, 128>>>(op, first, (uint64_t)per_thread, max_exponent, differing);
    const cudaError_t e = cudaGetLastError();
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}

// The units of a frame at S lanes per pixel, the pixels of its first n indices (-1: none), and whether
// it takes strips in a launch of that many patch units.
unsigned ktp_unit_count(int width, int height, int S, int strips) {
    return ktd::unit_count(width, height, S, false, strips != 0);
}
void ktp_frame_pixels(int width, int height, int strips, long long n, int* pixel) {
    for (long long i = 0; i < n; ++i) {
        int px = -1, py = -1;
        pixel[i] = ktd::frame_pixel((unsigned)i, width, height, strips != 0, px, py) ? py * width + px : -1;
    }
}
int ktp_take_strips(int width, int height, unsigned patch_units, unsigned warps) {
    return ktd::take_strips(width, height, patch_units, warps) ? 1 : 0;
}

}  // extern "C"
