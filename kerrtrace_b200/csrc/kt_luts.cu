// kt_luts.cu — the two lookup tables generated on the device.
//
// The same tables as the host generators (kt_generate_blackbody_lut, kt_generate_disk_lut in
// kt_host.cpp, which follow src/renderer/blackbody.rs:6-124 and src/renderer/utils.rs:11-52,
// 172-201), written into device memory on the caller's stream.
// This file is compiled without fast math: expm1f, expf, logf, acosf, cosf, cbrtf and sqrtf are
// CUDA's accurate versions, so the tables agree with the host ones to a few ulp (they are not
// bit-equal: CUDA's and glibc's libm round differently in the last place).
#include <cuda_runtime.h>
#include <stdint.h>

#include "kt_internal.h"

namespace ktd {

namespace {

// One lobe of the piecewise-Gaussian fit to the CIE 1931 matching functions.
__device__ float cmf_lobe_d(float x, float alpha, float mu, float s1, float s2) {
    const float sigma = x < mu ? s1 : s2;
    const float t = (x - mu) / sigma;
    return alpha * expf(-0.5f * t * t);
}

// Row ti: the linear-sRGB colour of a blackbody at temperature ti / (size - 1) x max_temp,
// integrated over the wavelength grid wl_start, wl_start + wl_step, ... (f32 accumulation, as the
// host grid) with the Planck law and the XYZ -> linear-sRGB matrix.
//
// What bounds it: latency, at the sizes in use (4096 rows x 35 wavelengths are two Planck terms per
// core).  A block takes kRows rows and kChunk wavelengths at a time: the matching functions are
// evaluated once per block, one thread per wavelength, the Planck terms one thread per (row,
// wavelength), and only the sums, whose order fixes the table's bits, run in sequence, one thread
// per row and channel.  With one thread per row doing all of it (7 exponentials of the matching
// functions per term), back to back: 4096 rows x 35 wavelengths 30.9 us, now 7.3; 16384 x 341 252 us,
// now 46; 100 x 1134 854 us, now 82.  Both table kernels come up under the one ahead and wait for it
// only before they store (launch_early): the two tables of 4096 rows, in turn, 11.3 -> 7.1 us.
constexpr int kRows = 16, kChunk = 64, kLutThreads = 128;
__global__ void __launch_bounds__(kLutThreads) blackbody_lut_kernel(uint32_t size, float max_temp, float wl_start,
                                                                    int n_lambda, float wl_step,
                                                                    float4* __restrict__ out) {
    __shared__ float lambda[kChunk], cmf[3][kChunk], planck[kRows][kChunk + 1], sums[kRows][3];
    let_next_launch();
    const uint32_t row0 = blockIdx.x * kRows;
    const int tid = threadIdx.x;
    const int sum_row = tid / 3, ch = tid - 3 * sum_row;
    float acc = 0.0f;
    float l0 = wl_start;  // first wavelength of the chunk
    for (int i0 = 0; i0 < n_lambda; i0 += kChunk) {
        const int n = n_lambda - i0 < kChunk ? n_lambda - i0 : kChunk;
        if (tid < n) {
            float l = l0;
            for (int i = 0; i < tid; ++i) l += wl_step;
            lambda[tid] = l;
            cmf[0][tid] = cmf_lobe_d(l, 1.056f, 599.8f, 37.9f, 31.0f) + cmf_lobe_d(l, 0.362f, 442.0f, 16.0f, 26.7f) +
                          cmf_lobe_d(l, -0.065f, 501.1f, 20.4f, 26.2f);
            cmf[1][tid] = cmf_lobe_d(l, 0.821f, 568.8f, 46.9f, 40.5f) + cmf_lobe_d(l, 0.286f, 530.9f, 16.3f, 31.1f);
            cmf[2][tid] = cmf_lobe_d(l, 1.217f, 437.0f, 11.8f, 36.0f) + cmf_lobe_d(l, 0.681f, 459.0f, 26.2f, 13.8f);
        }
        __syncthreads();
        for (int k = tid; k < kRows * n; k += kLutThreads) {
            const int row = k / n, i = k - row * n;
            const uint32_t ti = row0 + row;
            const float t = (float)((double)ti / (double)(size - 1) * (double)max_temp);
            float inten = 0.0f;
            if (ti < size && t > 0.0f) {
                const float l = lambda[i];
                const float expo = 1.4388e7f / (l * t);
                if (!(expo > 80.0f)) {
                    const float l2 = l * l;
                    const float l5 = l * (l2 * l2);
                    inten = ((1.0f / l5) / expm1f(expo)) * 1e15f;
                }
            }
            planck[row][i] = inten;
        }
        __syncthreads();
        if (tid < 3 * kRows)
            for (int i = 0; i < n; ++i) acc += planck[sum_row][i] * cmf[ch][i];
        if (i0 + kChunk < n_lambda) {
            for (int i = 0; i < kChunk; ++i) l0 += wl_step;
            __syncthreads();
        }
    }
    if (tid < 3 * kRows) sums[sum_row][ch] = acc * wl_step;
    wait_for_stream();
    __syncthreads();
    const uint32_t ti = row0 + tid;
    if (tid >= kRows || ti >= size) return;
    const float t = (float)((double)ti / (double)(size - 1) * (double)max_temp);
    if (t == 0.0f) {
        out[ti] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        return;
    }
    const float xsum = sums[tid][0], ysum = sums[tid][1], zsum = sums[tid][2];
    out[ti] = make_float4(fmaf(3.240454f, xsum, fmaf(-1.5371385f, ysum, -0.4985314f * zsum)),
                          fmaf(-0.969266f, xsum, fmaf(1.8760108f, ysum, 0.041556f * zsum)),
                          fmaf(0.0556434f, xsum, fmaf(-0.2040259f, ysum, 1.0572252f * zsum)), 0.0f);
}

// Page-Thorne flux factor with the roots 2 cos(acos(-a)/3 - 2 pi k / 3) of x^3 - 3x + 2a = 0.
__device__ float nt_factor_d(float r, float a_norm, float r_isco, float inv_m) {
    if (r <= r_isco) return 0.0f;
    const float r_norm = r * inv_m;
    const float r_isco_norm = r_isco * inv_m;
    const float x = sqrtf(r_norm);
    const float x_ms = sqrtf(r_isco_norm);
    const float third = 1.0f / 3.0f;
    const float angle_base = acosf(-a_norm) * third;
    const float ang_step = 2.0943952f;
    const float roots[3] = {2.0f * cosf(angle_base), 2.0f * cosf(angle_base - ang_step),
                            2.0f * cosf(angle_base + ang_step)};
    float sum_log = 0.0f;
    for (int i = 0; i < 3; ++i) {
        const float xi = roots[i];
        const float den = xi * (xi - roots[(i + 1) % 3]) * (xi - roots[(i + 2) % 3]);
        if (den <= 0.0f) continue;
        const float coef = 3.0f * (xi - a_norm) * (xi - a_norm) / den;
        const float val = (x - xi) / (x_ms - xi);
        if (val > 0.0f) sum_log += coef * logf(val);
    }
    const float q = fmaf(1.5f * a_norm, -logf(x / x_ms), x - x_ms) - sum_log;
    const float geo = r_norm * fmaf(2.0f, a_norm, fmaf(r_norm, x, -(3.0f * x)));
    return fmaxf(q / geo, 0.0f);
}

// Row i: f^(1/4) of the flux factor at r_i = r_in + i / (size - 1) (r_out - r_in).
__global__ void disk_lut_kernel(uint32_t size, float a_norm, float inv_m, float r_in, float r_out,
                                float* __restrict__ out) {
    let_next_launch();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= size) return;
    const double ratio = (double)i / (double)(size - 1);
    const float r = (float)fma(ratio, (double)(r_out - r_in), (double)r_in);
    const float f = sqrtf(sqrtf(nt_factor_d(r, a_norm, r_in, inv_m)));
    wait_for_stream();
    out[i] = f;
}

}  // namespace

cudaError_t launch_blackbody_lut(uint32_t size, float max_temp, float wl_start, int n_lambda, float wl_step,
                                 float4* out, cudaStream_t st) {
    return launch_early(blackbody_lut_kernel, dim3((size + kRows - 1) / kRows), kLutThreads, 0, st, size, max_temp, wl_start,
                        n_lambda, wl_step, out);
}

cudaError_t launch_disk_lut(uint32_t size, float a_norm, float inv_m, float r_in, float r_out, float* out,
                            cudaStream_t st) {
    return launch_early(disk_lut_kernel, dim3((size + 127) / 128), 128, 0, st, size, a_norm, inv_m, r_in, r_out, out);
}

}  // namespace ktd
