// device_probe.cu — runs single device functions of the product on given operands.  TEST
// INFRASTRUCTURE ONLY: built from the product's headers with the flags of its kernels, so that
// functions which no entry point exposes by themselves can be compared with CUDA's own.
//
// Every launch is one thread per operand, in bounds by construction; the C functions take device
// pointers, run on the legacy stream and return the CUDA status after a synchronisation.
#include <cuda_runtime.h>
#include <stdint.h>

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

}  // namespace

extern "C" {

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

}  // extern "C"
