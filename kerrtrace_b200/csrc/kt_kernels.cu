// kt_kernels.cu — trace and post-process kernels for sm_100a.
//
// Built with -use_fast_math, the flag set the reference compiles kernel.cu with
// (config.yaml `cuda.use_fast_math: true`, src/renderer/init.rs:112-118), so that `/`, powf and
// expf lower to the same instructions as in the reference.
//
// Trace kernels (replace trace_kernel, cuda/kernel.cu:88-142):
//   trace_plain_kernel      one thread per pixel on a 2D grid of block_dim tiles; each thread
//                           runs its spp rays to completion through the attempt state machine.
//   trace_wavefront_kernel  warps take units of 32 rays (pixels x samples): persistent warps, the first
//                           unit by index and the others from a device work counter, or a warp
//                           per unit.
// Post kernels (replace bloom_horizontal / post_process, cuda/kernel.cu:144-251):
//   bloom_h_kernel          horizontal normalised Gaussian over tiles staged in pairs of rows
//   post_v_kernel           vertical Gaussian over tiles staged in pairs of columns + composite,
//                           ACES, sRGB OETF, 0x00RRGGBB pack
//   tonemap_kernel          tone map alone (bloom inactive)
// kt_post_fused runs both passes over a bloom buffer that the context owns, laid out as the vertical
// pass stages it.  The post kernels produce the reference's bits: same tap order, weights, division
// and tone-map expressions.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "kt_internal.h"
#include "kt_ray.cuh"

namespace ktd {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWavefrontBlock = 128;

// ---- work counters (counting kernels only) -----------------------------------------------
__device__ __forceinline__ void add_tally(unsigned long long* ctr, uint64_t rays, const Tally& t) {
    atomicAdd(ctr + 0, (unsigned long long)rays);
    atomicAdd(ctr + 1, (unsigned long long)t.steps);
    atomicAdd(ctr + 2, (unsigned long long)t.attempts);
    atomicAdd(ctr + 3, (unsigned long long)t.rhs);
    atomicAdd(ctr + 4, (unsigned long long)t.frozen);
    atomicAdd(ctr + 5, (unsigned long long)t.fp64);
}
__device__ __forceinline__ void tally_ray(Tally& acc, const Tally& ray) {
    acc.steps += ray.steps;
    acc.attempts += ray.attempts;
    acc.rhs += ray.rhs;
    acc.frozen += ray.frozen ? 1u : 0u;
    acc.fp64 += ray.fp64;
}
// First shaded disk hit of sample 0 of a pixel (counting kernels, when aux is given).
__device__ __forceinline__ void write_aux(float4* aux, size_t idx, const Tally& t) {
    if (aux) aux[idx] = make_float4(t.first_r, t.first_g, t.first_T, (float)t.hits);
}

// Runs one ray per lane to completion and adds its colour to acc (A: float, or the ray's colour
// type).  active: the lane has a ray; later_sample: see ray_start; TOGETHER: see run_rays.
template <class R, int MODE, bool COUNT, bool TOGETHER, class A>
__device__ __forceinline__ void run_ray(bool active, int px, int py, int smp, const Scene& sc,
                                        const Camera& cam, uint32_t* err, A acc[3], Tally& total, float4* aux,
                                        bool later_sample = false) {
    RayRun<R> ry;
    Tally tl;
    tl.clear();
    bool run = false;
    if (active) {
        float dir[3];
        pixel_ray<MODE>(px, py, smp, sc, cam, dir);
        run = start(ry, cam, dir, sc, later_sample);
    }
    run_rays<MODE, COUNT, TOGETHER>(run, ry, sc, err, tl);
    if (!active) return;
    acc[0] += ry.col[0];
    acc[1] += ry.col[1];
    acc[2] += ry.col[2];
    if (COUNT) {
        tally_ray(total, tl);
        if (smp == 0) write_aux(aux, (size_t)py * sc.width + px, tl);
    }
}

// Work unit -> pixel.  Units run over 16-row bands, 16-column tiles inside a band, row-major
// inside a tile, so 32 consecutive units form a 16x2 patch (the footprint of one warp of the
// reference's 16x16 blocks).  Exact bijection onto [0, W) x [0, H), partial tiles included.
__device__ __forceinline__ void unit_to_pixel(unsigned u, int W, int H, int& px, int& py) {
    const unsigned band_px = (unsigned)W * 16u;
    const unsigned band = u / band_px;
    const unsigned rem = u - band * band_px;
    const int row0 = (int)band * 16;
    const int hb = min(16, H - row0);
    const unsigned tile_px = 16u * (unsigned)hb;
    const unsigned tile = rem / tile_px;
    const unsigned rem2 = rem - tile * tile_px;
    const int col0 = (int)tile * 16;
    const int wt = min(16, W - col0);
    py = row0 + (int)(rem2 / (unsigned)wt);
    px = col0 + (int)(rem2 % (unsigned)wt);
}

// ---- long-rays-first pixel order -----------------------------------------------------------
// A ray that passes close to a spherical photon orbit winds around the hole about ln(1/delta)
// times before it falls in or escapes, and takes several times the average step count.  Traced
// last, such rays leave single latency-bound warps running after the rest of the frame is done.
// The Kerr constants of motion of the initial state (E = -p_t, the angular momentum about the
// spin axis L = z p_x - x p_z, the Carter constant Q, with p_theta from the spheroidal
// coordinates of the Kerr-Schild point) fix the radial potential
//   R(r) = (E (r^2 + a^2) - a L)^2 - (r^2 - 2 M r + a^2) ((L - a E)^2 + Q),
// whose local minimum outside the horizon is close to 0 exactly for those rays.  The rank kernel
// marks pixels with |R(r_min)| < kHotThreshold E^2 r_min^4 (0.2% to 4% of a frame) and writes
// a permutation of the pixels: the marked ones first, then the rest in tile order.  The tracers
// read it when the tuning's order is 1.  Per-pixel results do not depend on the order.
constexpr float kHotThreshold = 0.1f;

__device__ __forceinline__ bool predicted_long(const Scene& sc, const Camera& cam, const float dir[3]) {
    RayRun<float> ry;
    ray_start<float>(ry, cam, dir, sc);
    const float a = sc.a, M = sc.M;
    const float x = ry.s[0], y = ry.s[1], z = ry.s[2];
    const float px = ry.s[3], py = ry.s[4], pz = ry.s[5];
    const float E = -ry.pt, E2 = E * E;
    const float L = z * px - x * pz;
    const float r = ks_radius<float>(x, y, z, sc.aa);
    const float ct = __fdividef(y, r);
    const float st2 = fmaxf(1.0f - ct * ct, 1e-12f);
    const float st = sqrtf(st2);
    const float pth = __fdividef(ct, st) * (x * px + z * pz) - r * st * py;
    const float Q = pth * pth + ct * ct * (__fdividef(L * L, st2) - a * a * E2);
    const float K = (L - a * E) * (L - a * E) + Q;
    const float B = a * (a * E - L);
    const float c2 = 2.0f * E * B - K;
    // Newton on R'(r) = 4 E^2 r^3 + 2 c2 r + 2 M K from the right of its largest root, where R'
    // is increasing and convex: the iterates decrease monotonically onto the root
    float rr = fmaxf(5.0f * M, sqrtf(__fdividef(fabsf(K), E2)));
#pragma unroll 1
    for (int it = 0; it < 16; ++it) {
        const float d1 = 4.0f * E2 * rr * rr * rr + 2.0f * c2 * rr + 2.0f * M * K;
        const float d2 = 12.0f * E2 * rr * rr + 2.0f * c2;
        if (!(d2 > 0.0f)) break;
        rr -= __fdividef(d1, d2);
    }
    const float r2 = rr * rr, r4 = r2 * r2;
    const float Rm = E2 * r4 + c2 * r2 + 2.0f * M * K * rr + B * B - a * a * K;
    return rr > sc.rh && fabsf(Rm) < kHotThreshold * E2 * r4;
}

// order[0], order[1]: marked / unmarked pixel counts; order[kOrderHeader + i]: pixel index
// py * width + px of work unit i.  Units are written in warp-sized runs (a 16x2 patch of the
// tile order, compacted): marked runs from the front, unmarked runs from the back.
__device__ __forceinline__ void ordered_pixel(unsigned u, unsigned n, const unsigned* order, unsigned n_hot,
                                              int W, int& px, int& py) {
    const unsigned* list = order + kOrderHeader;
    const unsigned idx = u < n_hot ? list[u] : list[n - 1u - (u - n_hot)];
    py = (int)(idx / (unsigned)W);
    px = (int)(idx - (unsigned)py * (unsigned)W);
}

template <int MODE>
__global__ void __launch_bounds__(256) rank_pixels_kernel(const Scene sc, const Camera cam,
                                                          unsigned* __restrict__ order) {
    const unsigned n = (unsigned)sc.width * (unsigned)sc.height;
    const unsigned u = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const bool valid = u < n;
    bool hot = false;
    unsigned idx = 0;
    if (valid) {
        int px, py;
        unit_to_pixel(u, sc.width, sc.height, px, py);
        idx = (unsigned)py * (unsigned)sc.width + (unsigned)px;
        float dir[3];
        pixel_ray<MODE>(px, py, 0, sc, cam, dir);
        hot = predicted_long(sc, cam, dir);
    }
    const unsigned hm = __ballot_sync(kFull, valid && hot);
    const unsigned cm = __ballot_sync(kFull, valid && !hot);
    unsigned hb = 0, cb = 0;
    if (lane == 0) {
        if (hm) hb = atomicAdd(order + 0, (unsigned)__popc(hm));
        if (cm) cb = atomicAdd(order + 1, (unsigned)__popc(cm));
    }
    hb = __shfl_sync(kFull, hb, 0);
    cb = __shfl_sync(kFull, cb, 0);
    const unsigned lt = (1u << lane) - 1u;
    unsigned* list = order + kOrderHeader;
    if (valid) {
        if (hot)
            list[hb + (unsigned)__popc(hm & lt)] = idx;
        else
            list[n - 1u - (cb + (unsigned)__popc(cm & lt))] = idx;
    }
}

// Resident 256-thread blocks per SM asked of the compiler for the plain kernel: two for the
// FP32 and mixed paths (at most 128 registers per thread, 16 warps per SM), one for FP64.
// Blocks of at most 128 threads can also ask for 5 or 6 resident blocks (at most 102 or 85
// registers: 20 or 24 warps per SM), a choice of the tuning (blocks_per_sm) for FP32 and mixed,
// and FP64 for 3 or 4 (at most 170 or 128 registers, with some spills: 12 or 16 warps per SM
// instead of 8).
template <class R> struct PlainMinBlocks { static constexpr int v = 2; };
template <> struct PlainMinBlocks<double> { static constexpr int v = 1; };

template <class R, int MODE, bool COUNT, int MAXT, int MINB = (MAXT == 256 ? PlainMinBlocks<R>::v : 1)>
__global__ void __launch_bounds__(MAXT, MINB)
    trace_plain_kernel(const __grid_constant__ Scene sc, const Camera cam,
                                                           float4* __restrict__ hdr,
                                                           uint32_t* __restrict__ err,
                                                           unsigned long long* __restrict__ ctr,
                                                           float4* __restrict__ aux,
                                                           const unsigned* __restrict__ order) {
    int px, py;
    if (order) {  // 1D launch over the ranked work units
        const unsigned n = (unsigned)sc.width * (unsigned)sc.height;
        const unsigned u = blockIdx.x * (blockDim.x * blockDim.y) + threadIdx.y * blockDim.x + threadIdx.x;
        if (u >= n) return;
        ordered_pixel(u, n, order, order[0], sc.width, px, py);
    } else {
        px = blockIdx.x * blockDim.x + threadIdx.x;
        py = blockIdx.y * blockDim.y + threadIdx.y;
        if (px >= sc.width || py >= sc.height) return;
    }
    float acc[3] = {0.0f, 0.0f, 0.0f};
    const int pix = py * sc.width + px;
    if (sc.accum && sc.sample_first > 0) {  // progressive: continue the running sum
        const float4 a = sc.accum[pix];
        acc[0] = a.x;
        acc[1] = a.y;
        acc[2] = a.z;
    }
    Tally total;
    total.clear();
    const int s_end = sc.sample_first + sc.spp;
    for (int smp = sc.sample_first; smp < s_end; ++smp)
        run_ray<R, MODE, COUNT, false>(true, px, py, smp, sc, cam, err, acc, total, aux);
    if (sc.accum) sc.accum[pix] = make_float4(acc[0], acc[1], acc[2], (float)s_end);
    const float fs = sc.final_scale;
    hdr[pix] = make_float4(acc[0] * fs, acc[1] * fs, acc[2] * fs, 1.0f);
    if (COUNT) add_tally(ctr, (uint64_t)sc.spp, total);
}

// Persistent tracer.  A warp takes units of P = 32 / S pixels and gives each pixel S lanes, one per
// sample (S = samples_in_parallel(spp); 1 at spp 1), so that the rays of a warp start together
// and, with S > 1, come from a smaller patch of the frame.  Its first unit is its own index in
// the grid, the others come from a device counter, so a frame of no more units than warps
// needs neither the counter nor its reset.  The samples of a pixel are added in sample order
// (shuffles over its lanes), as the plain kernel's loop adds them: the same bits.
//
// What bounds it: the FP32 (FP64) pipes, as the plain kernel; lanes idle only while the last rays
// of their own unit finish.  An earlier form refilled single lanes from the counter as their
// rays ended: each refill ran the start-up code (ray set-up, first tolerance, first right-hand
// side) for one lane of 32, which cost more than the idle lanes it filled.  Against it (trace and
// post, default tuning; with the later steps in it): 1920x1080 reference 3.58 -> 2.21 ms (trace),
// 960x540 FP64 6.27 -> 2.99, 1024^2 mixed 2.62 -> 1.09, two frames of 2100x900 at 4 samples 15.6 -> 7.13;
// 96x64 at 2 samples 0.279 -> 0.075, where a pixel's samples used to run one after the other on one lane.
template <class R, int MODE, bool COUNT, int MINB, bool TOGETHER, bool STRIPS>
__global__ void __launch_bounds__(kWavefrontBlock, MINB)
    trace_wavefront_kernel(const __grid_constant__ Scene sc, const Camera cam, float4* __restrict__ hdr,
                           uint32_t* __restrict__ err, unsigned* __restrict__ queue,
                           unsigned long long* __restrict__ ctr, float4* __restrict__ aux, int S,
                           const unsigned* __restrict__ order) {
    if (TOGETHER) wait_for_stream();
    const int lane = threadIdx.x & 31;
    const int slot = lane / S, sub = lane - slot * S;
    const unsigned P = 32u / (unsigned)S;
    const unsigned n_px = (unsigned)sc.width * (unsigned)sc.height;
    const unsigned units = unit_count(sc.width, sc.height, S, order != nullptr, STRIPS);
    const unsigned n_hot = order ? order[0] : 0u;
    const unsigned n_warps = gridDim.x * (kWavefrontBlock / 32);
    Tally total;
    total.clear();
    uint64_t rays = 0;

    for (unsigned u = blockIdx.x * (kWavefrontBlock / 32) + (threadIdx.x >> 5); u < units;) {
        const unsigned idx = u * P + (unsigned)slot;
        int px = 0, py = 0;
        bool valid = (unsigned)slot < P;
        if (order) {
            valid = valid && idx < n_px;
            if (valid) ordered_pixel(idx, n_px, order, n_hot, sc.width, px, py);
        } else {
            valid = valid && frame_pixel(idx, sc.width, sc.height, STRIPS, px, py);
        }
        float acc[3] = {0.0f, 0.0f, 0.0f};
        for (int s0 = 0; s0 < sc.spp; s0 += S) {
            decltype(RayRun<R>::tau) col[3] = {0, 0, 0};
            const bool has_sample = valid && s0 + sub < sc.spp;
            run_ray<R, MODE, COUNT, TOGETHER>(has_sample, px, py, s0 + sub, sc, cam, err, col, total, aux, s0 + sub > 0);
            if (COUNT && has_sample) ++rays;
            if (S == 1) {
#pragma unroll
                for (int c = 0; c < 3; ++c) acc[c] += col[c];
            } else {
                const int last = min(S, sc.spp - s0);
                for (int i = 0; i < last; ++i) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) acc[c] += __shfl_sync(kFull, col[c], min(slot * S + i, 31));
                }
            }
        }
        if (valid && sub == 0) {
            const float fs = sc.final_scale;
            hdr[py * sc.width + px] = make_float4(acc[0] * fs, acc[1] * fs, acc[2] * fs, 1.0f);
        }
        if (units <= n_warps) break;
        if (lane == 0) u = n_warps + atomicAdd(queue, 1u);
        u = __shfl_sync(kFull, u, 0);
    }
    if (COUNT) add_tally(ctr, rays, total);
}

// ---- launch -------------------------------------------------------------------------------
// Resident blocks per SM requested from the compiler (which caps registers per thread at
// 65536 / (128 * MINB)): the default per arithmetic type, and the variants the autotuner may
// pick for the FP32 reference-semantics kernel.
template <class R> struct WaveDefaults { static constexpr int minb = 4; };
template <> struct WaveDefaults<double> { static constexpr int minb = 2; };
template <> struct WaveDefaults<Mixed> { static constexpr int minb = 4; };

template <class R, int MODE, bool COUNT>
static cudaError_t launch_plain(const Scene& sc, const Camera& cam, float4* hdr, uint32_t* err,
                                unsigned long long* ctr, float4* aux, int bx, int by, int minb,
                                const unsigned* order, cudaStream_t st) {
    const dim3 block(bx, by);
    const unsigned n = (unsigned)sc.width * (unsigned)sc.height, per = (unsigned)(bx * by);
    const dim3 grid = order ? dim3((n + per - 1) / per)
                            : dim3((sc.width + bx - 1) / bx, (sc.height + by - 1) / by);
    if constexpr (std::is_same<R, double>::value) {
        if (bx * by <= 128 && minb == 3) {
            trace_plain_kernel<R, MODE, COUNT, 128, 3><<<grid, block, 0, st>>>(sc, cam, hdr, err, ctr, aux, order);
            return cudaGetLastError();
        }
        if (bx * by <= 128 && minb == 4) {
            trace_plain_kernel<R, MODE, COUNT, 128, 4><<<grid, block, 0, st>>>(sc, cam, hdr, err, ctr, aux, order);
            return cudaGetLastError();
        }
    } else {
        if (bx * by <= 128 && minb == 5) {
            trace_plain_kernel<R, MODE, COUNT, 128, 5><<<grid, block, 0, st>>>(sc, cam, hdr, err, ctr, aux, order);
            return cudaGetLastError();
        }
        if (bx * by <= 128 && minb == 6) {
            trace_plain_kernel<R, MODE, COUNT, 128, 6><<<grid, block, 0, st>>>(sc, cam, hdr, err, ctr, aux, order);
            return cudaGetLastError();
        }
    }
    if (bx * by <= 256)
        trace_plain_kernel<R, MODE, COUNT, 256><<<grid, block, 0, st>>>(sc, cam, hdr, err, ctr, aux, order);
    else
        trace_plain_kernel<R, MODE, COUNT, 1024><<<grid, block, 0, st>>>(sc, cam, hdr, err, ctr, aux, order);
    return cudaGetLastError();
}

template <class R, int MODE, bool COUNT, int MINB>
static cudaError_t launch_wave_minb(const Scene& sc, const Camera& cam, float4* hdr, uint32_t* err,
                                    unsigned* queue, unsigned long long* ctr, float4* aux, const unsigned* order,
                                    cudaStream_t st) {
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    constexpr unsigned kWarps = kWavefrontBlock / 32;
    const int S = samples_in_parallel(sc.spp);
    const unsigned resident = (unsigned)(sms * MINB);
    const bool ordered = order != nullptr;
    constexpr bool kDefaultShape = !COUNT && MINB == WaveDefaults<R>::minb;  // the others keep the patches
    const bool strips = kDefaultShape && !ordered &&
                        take_strips(sc.width, sc.height, unit_count(sc.width, sc.height, S, false, false), resident * kWarps);
    const unsigned units = unit_count(sc.width, sc.height, S, ordered, strips);
    const unsigned blocks = (units + kWarps - 1) / kWarps;
    // Stated physics in FP32 and FP64: a block per four units, not only the resident ones.  The
    // hardware's block scheduler then hands out the units and the warps of a block start
    // together, at the same place of a loop body (30 KB in FP64) that outgrows the nearer instruction
    // caches; persistent warps drift apart and the FP64 kernel waited for instructions 0.7
    // cycles per issue.  960x540 FP64 3.24 -> 2.99 ms, 1920x1080 6.58 -> 5.75, 400x300 x 3 samples 2.89 ->
    // 2.66; 1920x1080 FP32 2.16-2.36 -> 2.08.  The mixed and the reference trace gain nothing (1.088 ->
    // 1.097, 2.217 -> 2.227) and stay persistent, unless frozen rays are kept to the end (a switch for
    // timing): such a ray is a hundred times as long as the others of its unit, and blocks that come
    // up as others end fill the SMs better than warps that were dealt units before (1920x1080
    // 187 -> 152 ms; single lanes refilled from the counter took 183).
    constexpr bool kAllBlocks = MODE == 1 && !std::is_same<R, Mixed>::value;
    const unsigned grid = kAllBlocks || sc.keep_frozen || blocks < resident ? blocks : resident;
    if (units > grid * kWarps) {
        e = cudaMemsetAsync(queue, 0, sizeof(unsigned), st);
        if (e != cudaSuccess) return e;
    }
    // At most one unit per resident warp: the launch lasts as long as its longest rays, and the warp
    // that keeps its lanes in step issues fewer instructions for them (96x64 x 2 samples 78.3 -> 72.2
    // us, 256x256 at tolerance 1e-8 23.9 -> 23.3 ms).  With more units the vote and the register
    // moves around it cost more than they save (1920x1080 2.21 -> 2.37 ms).
    if constexpr (kDefaultShape) {
        if (strips) {
            trace_wavefront_kernel<R, MODE, COUNT, MINB, false, true>
                <<<grid, kWavefrontBlock, 0, st>>>(sc, cam, hdr, err, queue, ctr, aux, S, order);
            return cudaGetLastError();
        }
        if (units <= resident * kWarps) {
            if (order) {
                trace_wavefront_kernel<R, MODE, COUNT, MINB, true, false>
                    <<<grid, kWavefrontBlock, 0, st>>>(sc, cam, hdr, err, queue, ctr, aux, S, order);
                return cudaGetLastError();
            }
            return launch_early(trace_wavefront_kernel<R, MODE, COUNT, MINB, true, false>, dim3(grid), kWavefrontBlock, 0,
                                st, sc, cam, hdr, err, queue, ctr, aux, S, order);
        }
    }
    trace_wavefront_kernel<R, MODE, COUNT, MINB, false, false>
        <<<grid, kWavefrontBlock, 0, st>>>(sc, cam, hdr, err, queue, ctr, aux, S, order);
    return cudaGetLastError();
}

template <class R, int MODE, bool COUNT>
static cudaError_t launch_wave(const Scene& sc, const Camera& cam, float4* hdr, uint32_t* err,
                               unsigned* queue, unsigned long long* ctr, float4* aux, const Tuning& tn,
                               const unsigned* order, cudaStream_t st) {
    if constexpr (std::is_same<R, float>::value && MODE == 0 && !COUNT) {
        switch (tn.blocks_per_sm) {
            case 3: return launch_wave_minb<R, MODE, COUNT, 3>(sc, cam, hdr, err, queue, ctr, aux, order, st);
            case 5: return launch_wave_minb<R, MODE, COUNT, 5>(sc, cam, hdr, err, queue, ctr, aux, order, st);
            case 6: return launch_wave_minb<R, MODE, COUNT, 6>(sc, cam, hdr, err, queue, ctr, aux, order, st);
            default: break;
        }
    }
    return launch_wave_minb<R, MODE, COUNT, WaveDefaults<R>::minb>(sc, cam, hdr, err, queue, ctr, aux, order, st);
}

template <class R, int MODE>
static cudaError_t launch_typed(const Scene& sc, const Camera& cam, int schedule, float4* hdr,
                                uint32_t* err, unsigned* queue, unsigned long long* ctr, float4* aux,
                                const Tuning& tn, int bx, int by, unsigned* order, cudaStream_t st) {
    if (order) {
        const unsigned n = (unsigned)sc.width * (unsigned)sc.height;
        cudaError_t e = cudaMemsetAsync(order, 0, 2 * sizeof(unsigned), st);
        if (e != cudaSuccess) return e;
        rank_pixels_kernel<MODE><<<(n + 255) / 256, 256, 0, st>>>(sc, cam, order);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if (schedule == 0)
        return ctr ? launch_plain<R, MODE, true>(sc, cam, hdr, err, ctr, aux, bx, by, tn.blocks_per_sm, order, st)
                   : launch_plain<R, MODE, false>(sc, cam, hdr, err, ctr, aux, bx, by, tn.blocks_per_sm, order, st);
    return ctr ? launch_wave<R, MODE, true>(sc, cam, hdr, err, queue, ctr, aux, tn, order, st)
               : launch_wave<R, MODE, false>(sc, cam, hdr, err, queue, ctr, aux, tn, order, st);
}

cudaError_t launch_trace(const Scene& sc, const Camera& cam, int schedule, float4* hdr,
                         uint32_t* err, unsigned* queue, unsigned long long* ctr, float4* aux,
                         const Tuning& tn, int bx, int by, unsigned* order, cudaStream_t st) {
    if (sc.width <= 0 || sc.height <= 0) return cudaSuccess;
    if (sc.precision == 2) return launch_typed<double, 1>(sc, cam, schedule, hdr, err, queue, ctr, aux, tn, bx, by, order, st);
    if (sc.precision == 1) return launch_typed<Mixed, 1>(sc, cam, schedule, hdr, err, queue, ctr, aux, tn, bx, by, order, st);
    if (sc.mode == 1) return launch_typed<float, 1>(sc, cam, schedule, hdr, err, queue, ctr, aux, tn, bx, by, order, st);
    return launch_typed<float, 0>(sc, cam, schedule, hdr, err, queue, ctr, aux, tn, bx, by, order, st);
}

// ---- batched renders -----------------------------------------------------------------------
template <class R, int MODE, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT == 256 ? PlainMinBlocks<R>::v : 1)
    trace_batch_kernel(const __grid_constant__ BatchTable bt) {
    const int b = blockIdx.x;
    int j = 0;
    while (j + 1 < bt.n && b >= bt.job[j + 1].tile_begin) ++j;
    const BatchJob& jb = bt.job[j];
    const Scene& sc = jb.sc;
    const int t = b - jb.tile_begin;
    const int ty = t / jb.tiles_x, tx = t - ty * jb.tiles_x;
    const int px = tx * (int)blockDim.x + (int)threadIdx.x;
    const int py = ty * (int)blockDim.y + (int)threadIdx.y;
    if (px >= sc.width || py >= sc.height) return;
    float acc[3] = {0.0f, 0.0f, 0.0f};
    Tally total;
    total.clear();
    for (int smp = 0; smp < sc.spp; ++smp)
        run_ray<R, MODE, false, false>(true, px, py, smp, sc, jb.cam, jb.err, acc, total, nullptr);
    const float fs = sc.final_scale;
    jb.hdr[py * sc.width + px] = make_float4(acc[0] * fs, acc[1] * fs, acc[2] * fs, 1.0f);
}

template <class R, int MODE>
static cudaError_t launch_batch_typed(const BatchTable& bt, int bx, int by, cudaStream_t st) {
    if (bx * by <= 256)
        trace_batch_kernel<R, MODE, 256><<<bt.total_tiles, dim3(bx, by), 0, st>>>(bt);
    else
        trace_batch_kernel<R, MODE, 1024><<<bt.total_tiles, dim3(bx, by), 0, st>>>(bt);
    return cudaGetLastError();
}

cudaError_t launch_batch(const BatchTable& bt, int bx, int by, cudaStream_t st) {
    if (bt.n <= 0 || bt.total_tiles <= 0) return cudaSuccess;
    const Scene& s0 = bt.job[0].sc;
    if (s0.precision == 2) return launch_batch_typed<double, 1>(bt, bx, by, st);
    if (s0.precision == 1) return launch_batch_typed<Mixed, 1>(bt, bx, by, st);
    if (s0.mode == 1) return launch_batch_typed<float, 1>(bt, bx, by, st);
    return launch_batch_typed<float, 0>(bt, bx, by, st);
}

// Persistent batched trace.  Every job is cut into units of 32 pixels (frame_pixel's order, so a
// unit is an 8x4 patch of one frame); job j owns units [unit_begin, unit_begin of j + 1).  A
// warp's first unit is its own index in the grid, the others come from a single device counter
// over all jobs, so the 32 rays of a warp always share one scene and its parameters stay uniform
// constant-bank loads, and an SM never waits for a whole block: each warp moves on as soon as
// its own unit is done.  Per-pixel arithmetic is the plain kernel's (run_ray).
//
// Bound by the FP32 pipe; lanes idle while the longest ray of their unit finishes, and a square
// patch holds rays more alike than one of 16x2: 64 renders of 128x128 to 960x540 15.75 -> 15.45
// ms, 64 up to 400x225 3.01 -> 2.95.  A batch of one unit per warp at most lasts as long as its
// longest ray, and takes the loop that keeps a warp's lanes in step (TOGETHER): two renders of
// 100 columns 130 -> 104 us, five of up to 160 181 -> 130.  In FP64 every unit gets its warp at the launch
// (64 renders of 64x64 to 480x270: 12.16 -> 11.24 ms; stated FP32 3.27 -> 3.37, so it does not).
template <class R, int MODE, int MINB, bool TOGETHER>
__global__ void __launch_bounds__(kWavefrontBlock, MINB)
    trace_batch_persistent_kernel(const __grid_constant__ BatchTable bt, unsigned* __restrict__ counter) {
    const int lane = threadIdx.x & 31;
    const unsigned n_warps = gridDim.x * (kWavefrontBlock / 32);
    for (unsigned u = blockIdx.x * (kWavefrontBlock / 32) + (threadIdx.x >> 5); u < bt.total_units;) {
        int lo = 0, hi = bt.n - 1;  // last job whose first unit is <= u
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (bt.job[mid].unit_begin <= u) lo = mid; else hi = mid - 1;
        }
        const BatchJob& jb = bt.job[lo];
        const Scene& sc = jb.sc;
        int px, py;
        const bool valid = frame_pixel((u - jb.unit_begin) * 32u + (unsigned)lane, sc.width, sc.height, jb.strips != 0, px, py);
        float acc[3] = {0.0f, 0.0f, 0.0f};
        Tally total;
        total.clear();
        for (int smp = 0; smp < sc.spp; ++smp)
            run_ray<R, MODE, false, TOGETHER>(valid, px, py, smp, sc, jb.cam, jb.err, acc, total, nullptr);
        if (valid) {
            const float fs = sc.final_scale;
            jb.hdr[py * sc.width + px] = make_float4(acc[0] * fs, acc[1] * fs, acc[2] * fs, 1.0f);
        }
        if (bt.total_units <= n_warps) break;
        if (lane == 0) u = n_warps + atomicAdd(counter, 1u);
        u = __shfl_sync(kFull, u, 0);
    }
}

template <class R, int MODE, int MINB>
static cudaError_t launch_batch_persistent_minb(const BatchTable& bt, unsigned* counter, cudaStream_t st) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, trace_batch_persistent_kernel<R, MODE, MINB, false>,
                                                           kWavefrontBlock, 0)) != cudaSuccess)
        return e;
    if (per_sm < 1) per_sm = 1;
    const unsigned warps = (unsigned)(sms * per_sm) * (kWavefrontBlock / 32);
    if (bt.total_units <= warps) {
        const unsigned blocks = (bt.total_units + kWavefrontBlock / 32 - 1) / (kWavefrontBlock / 32);
        trace_batch_persistent_kernel<R, MODE, MINB, true><<<blocks, kWavefrontBlock, 0, st>>>(bt, counter);
        return cudaGetLastError();
    }
    if (std::is_same<R, double>::value) {  // a block per four units, as the single frame (launch_wave_minb)
        const unsigned blocks = (bt.total_units + kWavefrontBlock / 32 - 1) / (kWavefrontBlock / 32);
        trace_batch_persistent_kernel<R, MODE, MINB, false><<<blocks, kWavefrontBlock, 0, st>>>(bt, counter);
        return cudaGetLastError();
    }
    if ((e = cudaMemsetAsync(counter, 0, sizeof(unsigned), st)) != cudaSuccess) return e;
    trace_batch_persistent_kernel<R, MODE, MINB, false><<<sms * per_sm, kWavefrontBlock, 0, st>>>(bt, counter);
    return cudaGetLastError();
}

cudaError_t launch_batch_persistent(const BatchTable& bt, int blocks_per_sm, unsigned* counter, cudaStream_t st) {
    if (bt.n <= 0 || bt.total_units == 0) return cudaSuccess;
    const Scene& s0 = bt.job[0].sc;
    if (s0.precision == 2) return launch_batch_persistent_minb<double, 1, 2>(bt, counter, st);
    if (s0.precision == 1) return launch_batch_persistent_minb<Mixed, 1, 4>(bt, counter, st);
    if (s0.mode == 1) return launch_batch_persistent_minb<float, 1, 4>(bt, counter, st);
    switch (blocks_per_sm) {
        case 5: return launch_batch_persistent_minb<float, 0, 5>(bt, counter, st);
        case 6: return launch_batch_persistent_minb<float, 0, 6>(bt, counter, st);
        default: return launch_batch_persistent_minb<float, 0, 4>(bt, counter, st);
    }
}

// ---- image comparison (the autotuner's bit-identity filter) ---------------------------------
__global__ void __launch_bounds__(256) count_mismatch_kernel(const uint4* __restrict__ a, const uint4* __restrict__ b,
                                                             size_t n, unsigned long long* __restrict__ out) {
    unsigned long long local = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const uint4 x = __ldg(a + i), y = __ldg(b + i);
        local += (x.x != y.x || x.y != y.y || x.z != y.z || x.w != y.w) ? 1u : 0u;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(kFull, local, o);
    if ((threadIdx.x & 31) == 0 && local) atomicAdd(out, local);
}

cudaError_t launch_count_mismatch(const void* a, const void* b, size_t n16, unsigned long long* out, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(unsigned long long), st);
    if (e != cudaSuccess || n16 == 0) return e;
    int dev = 0, sms = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    const size_t want = (n16 + 255) / 256;
    const unsigned blocks = (unsigned)(want < (size_t)sms * 8 ? want : (size_t)sms * 8);
    count_mismatch_kernel<<<blocks, 256, 0, st>>>(static_cast<const uint4*>(a), static_cast<const uint4*>(b), n16, out);
    return cudaGetLastError();
}

// =========================================================================================
// Post-processing
// =========================================================================================

// Gaussian tap weight (cuda/kernel.cu:48-53).
__device__ __forceinline__ float tap_weight(int i, float sigma) {
    const float t = (float)i;
    const float den = 2.0f * sigma * sigma;
    return __expf(-(t * t) / den);
}

// ACES filmic fit (cuda/kernel.cu:17-29) and sRGB OETF (cuda/kernel.cu:30-43).
__device__ __forceinline__ float aces1(float x) {
    const float a = 2.51f, b = 0.03f, c = 2.43f, d = 0.59f, e = 0.14f;
    return (x * (a * x + b)) / (x * (c * x + d) + e);
}
__device__ __forceinline__ float srgb1(float x) {
    if (x <= 0.0031308f) return 12.92f * x;
    return 1.055f * powf(x, 0.4166666666666667f) - 0.055f;
}
// Nearest integer of saturate(v) x 255 in the low byte: adding 3 x 2^22 leaves no fraction bits, so the
// addition rounds as the conversion instruction does, on the FMA pipe instead of the conversion unit.
__device__ __forceinline__ uint32_t to_byte(float v) {
    return __float_as_uint(__fadd_rn(__fmul_rn(__saturatef(v), 255.0f), 12582912.0f));
}
__device__ __forceinline__ uint32_t tone_pack(float r, float g, float b) {
    const float mr = srgb1(aces1(r)), mg = srgb1(aces1(g)), mb = srgb1(aces1(b));
    // bytes b, g, r and the zero above r's
    return __byte_perm(__byte_perm(to_byte(mb), to_byte(mg), 0x0040), to_byte(mr), 0x5410);
}

// Bloom source (stated physics: only the part of the luminance above the threshold blooms).
__device__ __forceinline__ float4 bloom_source(float4 c, const PostParams& pp) {
    if (pp.mode != 1) return c;
    const float L = 0.2126f * c.x + 0.7152f * c.y + 0.0722f * c.z;
    const float k = L > pp.threshold ? (L - pp.threshold) / L : 0.0f;
    return make_float4(c.x * k, c.y * k, c.z * k, c.w);
}

// ---- separable Gaussian on pairs of lines -------------------------------------------------
// A blur line is a row (horizontal pass) or a column (vertical pass).  A block blurs kTPairs pairs of
// lines over kTPos positions: its sources are staged in shared memory with the two lines of a pair
// side by side, (r0, r1, g0, g1) and (b0, b1), so that one packed multiply-add (fma.f32x2) makes a
// tap of both lines.  Each thread makes kBJ consecutive outputs of one pair from one stream of
// kBJ + 2R values: value k feeds output j with weight w[k - j] (tap i = k - j - R), so every output
// still accumulates its taps in increasing i, the order of the reference's loop
// (cuda/kernel.cu:156-166, 199-209), with the same single multiply-adds, and gets the same bits.
// Taps outside the image multiply staged zeros, which leaves a sum as it is (the reference skips
// them).
//
// What bounds it: the FMA pipe (3 (2R + 1) multiply-adds per pixel and pass).  A packed multiply-add
// holds the pipe as long as two plain ones but takes one issue slot, so the loads of the taps, the
// staging and the tone map (as many instructions as the blur itself at R = 24) go out beside it; the
// plain multiply-adds of an earlier form competed with them for slots and kept the pipe 37% busy.
// 64 x 32-pixel tiles of 128 threads: 43 KB and 5 blocks per SM at R = 24, 7 blocks per SM and
// frame at 1920x1080 (1020 blocks: a 128-wide tile would leave some SMs 4 and some 3).  Both passes
// back to back (fused), their launches overlapped (launch_early): 1920x1080 R = 24 66.4 -> 41.1 us,
// 3840x2160 213 -> 159 us, 2100x900 R = 48 118 -> 66.4 us, 960x540 30.9 -> 16.1 us.  Without the
// overlap 1920x1080 takes 45.1 us, without the blur as well 31, without the staging 41: what is left
// beside the multiply-adds (18 us) is each block's chain of loads, tone map and stores with 16 to
// 20 warps per SM to cover it (FMA pipe 41 and 45% active, issue 36 and 45%; 3.0 and 2.0 cycles of
// waiting for loads per issue).
constexpr int kBJ = 8, kTPairs = 16, kTPos = 64, kTThreads = kTPairs * (kTPos / kBJ);
constexpr int kTWarps = kTThreads / 32;

struct PairTile {
    ulonglong2* rg;  // kTPairs x stride: (r0, r1), (g0, g1)
    uint64_t* b;     // kTPairs x stride: (b0, b1)
    uint64_t* w;     // 2R + 2: (w, w), the last one zero
    float* inv;      // kTPos: 1 / weight sum of the tile's positions
};
// odd strides: the 8 (16) lanes of a shared-memory phase read different 16 (8)-byte banks
__host__ __device__ constexpr int pair_stride(int R) { return (kTPos + 2 * R) | 1; }
__host__ __device__ constexpr size_t pair_smem(int R) {
    return (size_t)kTPairs * pair_stride(R) * 24 + (size_t)(2 * R + 2) * 8 + kTPos * sizeof(float);
}
__device__ __forceinline__ PairTile pair_tile(void* smem, int R) {
    PairTile t;
    t.rg = static_cast<ulonglong2*>(smem);
    t.b = reinterpret_cast<uint64_t*>(t.rg + kTPairs * pair_stride(R));
    t.w = t.b + kTPairs * pair_stride(R);
    t.inv = reinterpret_cast<float*>(t.w + 2 * R + 2);
    return t;
}

__device__ __forceinline__ void tap2(uint64_t (&acc)[3], const ulonglong2& rg, uint64_t b, uint64_t w) {
    acc[0] = fma2(rg.x, w, acc[0]);
    acc[1] = fma2(rg.y, w, acc[1]);
    acc[2] = fma2(b, w, acc[2]);
}

// kBJ outputs of one pair; rg, b: the thread's first source.
__device__ __forceinline__ void blur_pair(const ulonglong2* rg, const uint64_t* b, const uint64_t* w, int R,
                                          uint64_t (&acc)[kBJ][3]) {
#pragma unroll
    for (int j = 0; j < kBJ; ++j) acc[j][0] = acc[j][1] = acc[j][2] = 0;
    if (2 * R < kBJ - 1) {  // fewer taps than outputs: one output after the other
#pragma unroll
        for (int j = 0; j < kBJ; ++j)
            for (int i = 0; i <= 2 * R; ++i) tap2(acc[j], rg[j + i], b[j + i], w[i]);
        return;
    }
    // The last kBJ weights in registers, weight i in slot i mod kBJ: every use has a fixed slot in
    // the unrolled steps and nothing is shifted.
    uint64_t wr[kBJ];
#pragma unroll
    for (int i = 0; i < kBJ; ++i) wr[i] = w[i];
    // head: value k (< kBJ - 1) feeds outputs 0..k
#pragma unroll
    for (int k = 0; k < kBJ - 1; ++k) {
        const ulonglong2 c = rg[k];
        const uint64_t d = b[k];
#pragma unroll
        for (int j = 0; j <= k; ++j) tap2(acc[j], c, d, wr[k - j]);
    }
    // middle: value k (kBJ - 1 .. 2R) feeds every output, in rounds of kBJ steps and a short last one
    const int mid = 2 * R + 2 - kBJ;
    int k0 = kBJ - 1;
#pragma unroll 1
    for (; k0 + kBJ <= kBJ - 1 + mid; k0 += kBJ) {
#pragma unroll
        for (int s = 0; s < kBJ; ++s) {
            const ulonglong2 c = rg[k0 + s];
            const uint64_t d = b[k0 + s];
#pragma unroll
            for (int j = 0; j < kBJ; ++j) tap2(acc[j], c, d, wr[(kBJ - 1 + s - j) % kBJ]);
            wr[s] = w[k0 + s + 1];
        }
    }
#pragma unroll
    for (int s = 0; s < kBJ - 1; ++s) {
        if (k0 + s > 2 * R) break;
        const ulonglong2 c = rg[k0 + s];
        const uint64_t d = b[k0 + s];
#pragma unroll
        for (int j = 0; j < kBJ; ++j) tap2(acc[j], c, d, wr[(kBJ - 1 + s - j) % kBJ]);
        wr[s] = w[k0 + s + 1];
    }
    // tail: value 2R + t feeds outputs t..kBJ-1 with weights 2R - kBJ + 2 .. 2R
#pragma unroll
    for (int i = 0; i < kBJ - 1; ++i) wr[i] = w[2 * R + 2 - kBJ + i];
#pragma unroll
    for (int t = 1; t < kBJ; ++t) {
        const ulonglong2 c = rg[2 * R + t];
        const uint64_t d = b[2 * R + t];
#pragma unroll
        for (int j = t; j < kBJ; ++j) tap2(acc[j], c, d, wr[kBJ - 2 + t - j]);
    }
}

// Four values per lane of a row pair, 32 apart, into the staged tile; `left`: values from the lane's
// first to the end of the segment.
__device__ __forceinline__ void store_row_pair(float4 (&u)[4], float4 (&v)[4], ulonglong2* rg, uint64_t* b, int left,
                                               const PostParams& pp) {
    if (pp.mode == 1) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            u[q] = bloom_source(u[q], pp);
            v[q] = bloom_source(v[q], pp);
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (32 * q < left) {
            rg[32 * q] = make_ulonglong2(pack2(u[q].x, v[q].x), pack2(u[q].y, v[q].y));
            b[32 * q] = pack2(u[q].z, v[q].z);
        }
    }
}
__device__ __forceinline__ void load_row_pair(const float4* row, int W, float4 (&u)[4], float4 (&v)[4], int left) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (32 * q < left) {
            u[q] = load_behind_wait(row + 32 * q);
            v[q] = load_behind_wait(row + W + 32 * q);
        }
    }
}

// Asynchronous copies global -> shared (cp.async); the bytes past src_bytes are zero-filled and
// nothing is read when src_bytes is 0.  Both addresses are aligned to the size.
__device__ __forceinline__ void copy16_async(void* dst, const void* src, int src_bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void copy8_async(void* dst, const void* src, int src_bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void copy_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

__device__ __forceinline__ void copy4_async(void* dst, const void* src, int src_bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
}

// Starts the copies of the weight pairs and of the positions' reciprocal sums (`inv` of `n` entries,
// from position p0); complete after copy_async_wait_all and a barrier.
__device__ __forceinline__ void stage_tables(const PairTile& t, const PostParams& pp, const float* inv, int p0, int n,
                                             int tid) {
    for (int i = tid; i < 2 * pp.radius + 2; i += kTThreads) copy8_async(t.w + i, pp.weights + i, 8);
    if (tid < kTPos) copy4_async(t.inv + tid, inv + (p0 + tid < n ? p0 + tid : 0), p0 + tid < n ? 4 : 0);
}

// The bloom buffer of the fused post: per pair of columns one column of (r0, r1, g0, g1), and, behind
// them, one of (b0, b1): 12 bytes per pixel in the order in which the vertical pass stages it.
__host__ __device__ __forceinline__ size_t bloom_pairs(int width) { return ((size_t)width + 1) / 2; }
size_t post_scratch_bytes(int width, int height) { return bloom_pairs(width) * (size_t)height * 24; }

// Horizontal pass (bloom_horizontal, cuda/kernel.cu:144-173): a block makes 32 rows x 64 columns.  A
// warp holds the 16 row pairs of two 8-column chunks.  PAIRED writes the fused post's bloom
// buffer straight from registers (a thread's 8 columns are 4 column pairs, consecutive pairs of rows
// consecutive in memory); the row-major output goes back through shared memory for coalesced
// stores.
template <bool PAIRED>
__global__ void __launch_bounds__(kTThreads, 5) bloom_h_kernel(const PostParams pp, const float4* __restrict__ hdr,
                                                               float4* __restrict__ bloom) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int R = pp.radius, W = pp.width, H = pp.height;
    const int stride = pair_stride(R), segw = kTPos + 2 * R;
    const PairTile t = pair_tile(smem_raw, R);
    const int x0 = blockIdx.x * kTPos, y0 = blockIdx.y * (2 * kTPairs);
    const int tid = threadIdx.x;
    if (PAIRED) let_next_launch();
    stage_tables(t, pp, pp.inv_wsum_x, x0, W, tid);
    wait_for_stream();
    {
        // a warp takes 4 row pairs, 128 columns of one at a time: 8 loads in flight per lane
        const int warp = tid >> 5, lane = tid & 31;
        const bool inner = x0 >= R && x0 + kTPos + R <= W && y0 + 2 * kTPairs <= H;  // no source outside
        const float4* src = hdr + (ptrdiff_t)(y0 + 2 * warp) * W + (x0 - R + lane);
        ulonglong2* rg = t.rg + warp * stride + lane;
        uint64_t* b = t.b + warp * stride + lane;
        if (inner) {
            for (int p = warp; p < kTPairs; p += kTWarps) {
                for (int c0 = 0; c0 < segw; c0 += 128) {
                    float4 u[4], v[4];
                    load_row_pair(src + c0, W, u, v, segw - c0 - lane);
                    store_row_pair(u, v, rg + c0, b + c0, segw - c0 - lane, pp);
                }
                src += (size_t)2 * kTWarps * W;
                rg += kTWarps * stride;
                b += kTWarps * stride;
            }
        } else {
            for (int p = warp; p < kTPairs; p += kTWarps) {
                const int y = y0 + 2 * p;
                for (int c0 = 0; c0 < segw; c0 += 128) {
                    float4 u[4], v[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int c = c0 + 32 * q, x = x0 - R + lane + c;
                        const bool in = x >= 0 && x < W && lane + c < segw;
                        u[q] = in && y < H ? load_behind_wait(src + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                        v[q] = in && y + 1 < H ? load_behind_wait(src + W + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                    store_row_pair(u, v, rg + c0, b + c0, segw - c0 - lane, pp);
                }
                src += (size_t)2 * kTWarps * W;
                rg += kTWarps * stride;
                b += kTWarps * stride;
            }
        }
        copy_async_wait_all();
    }
    __syncthreads();
    const int p = tid & (kTPairs - 1), cb = (tid / kTPairs) * kBJ;
    uint64_t acc[kBJ][3];
    blur_pair(t.rg + p * stride + cb, t.b + p * stride + cb, t.w, R, acc);
    const int xs = x0 + cb, y = y0 + 2 * p;
    // over the sum of the in-image weights (cuda/kernel.cu:167-171, 210-214), whose reciprocal the
    // tables hold: the fast division is that product (no division where the sum is 0: they hold 1)
#pragma unroll
    for (int j = 0; j < kBJ; ++j) {
        const float s = t.inv[cb + j];
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[j][c] = mul2(acc[j][c], pack2(s, s));
    }
    if (PAIRED) {
        float4* rg = bloom;
        float2* b = reinterpret_cast<float2*>(bloom + bloom_pairs(W) * H);
#pragma unroll
        for (int j = 0; j < kBJ; j += 2) {
            if (xs + j >= W) break;
            const size_t at = (size_t)((xs + j) >> 1) * H + y;
            if (y < H) {
                rg[at] = make_float4(lo2(acc[j][0]), lo2(acc[j + 1][0]), lo2(acc[j][1]), lo2(acc[j + 1][1]));
                b[at] = make_float2(lo2(acc[j][2]), lo2(acc[j + 1][2]));
            }
            if (y + 1 < H) {
                rg[at + 1] = make_float4(hi2(acc[j][0]), hi2(acc[j + 1][0]), hi2(acc[j][1]), hi2(acc[j + 1][1]));
                b[at + 1] = make_float2(hi2(acc[j][2]), hi2(acc[j + 1][2]));
            }
        }
        return;
    }
    // 2 x kTPairs rows of kTPos float4 (odd stride): no more than the staged sources took
    __syncthreads();
    constexpr int ostride = kTPos + 1;
    float4* out = reinterpret_cast<float4*>(smem_raw);
    for (int half = 0; half < 2; ++half) {
#pragma unroll
        for (int j = 0; j < kBJ; ++j)
            out[p * ostride + cb + j] = half ? make_float4(hi2(acc[j][0]), hi2(acc[j][1]), hi2(acc[j][2]), 0.0f)
                                             : make_float4(lo2(acc[j][0]), lo2(acc[j][1]), lo2(acc[j][2]), 0.0f);
        __syncthreads();
        for (int i = tid; i < kTPairs * kTPos; i += kTThreads) {
            const int r = i / kTPos, c = i - r * kTPos;
            const int gy = y0 + 2 * r + half, gx = x0 + c;
            if (gy < H && gx < W) bloom[(size_t)gy * W + gx] = out[r * ostride + c];
        }
        __syncthreads();
    }
}

// Vertical pass + composite + ACES + sRGB + pack (post_process, cuda/kernel.cu:175-251): a block makes
// 32 columns x 64 rows; a warp holds the 16 column pairs of two 8-row chunks.  PAIRED stages the
// fused post's bloom buffer by cp.async; otherwise the row-major buffer of bloom_horizontal is
// paired on the way in.
template <bool PAIRED>
__global__ void __launch_bounds__(kTThreads, 4) post_v_kernel(const PostParams pp, const float4* __restrict__ hdr,
                                                              const float4* __restrict__ bloom,
                                                              uint32_t* __restrict__ image) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int R = pp.radius, W = pp.width, H = pp.height;
    const int stride = pair_stride(R), segw = kTPos + 2 * R;
    const PairTile t = pair_tile(smem_raw, R);
    const int x0 = blockIdx.x * (2 * kTPairs), y0 = blockIdx.y * kTPos;
    const int tid = threadIdx.x;
    stage_tables(t, pp, pp.inv_wsum_y, y0, H, tid);
    wait_for_stream();
    if (PAIRED) {
        const int warp = tid >> 5, lane = tid & 31;
        const size_t pairs = bloom_pairs(W);
        const float2* bl = reinterpret_cast<const float2*>(bloom + pairs * H);
        const bool inner = y0 >= R && y0 + kTPos + R <= H && x0 / 2 + kTPairs <= (int)pairs;
        ptrdiff_t at = (ptrdiff_t)(x0 / 2 + warp) * H + (y0 - R + lane);
        ulonglong2* rg = t.rg + warp * stride + lane;
        uint64_t* b = t.b + warp * stride + lane;
        for (int p = warp; p < kTPairs; p += kTWarps) {
            if (inner) {
#pragma unroll 4
                for (int c = 0; c < segw - lane; c += 32) {
                    copy16_async(rg + c, bloom + at + c, 16);
                    copy8_async(b + c, bl + at + c, 8);
                }
            } else {
                const bool line = x0 / 2 + p < (int)pairs;
                for (int c = 0; c < segw - lane; c += 32) {
                    const int y = y0 - R + lane + c;
                    const bool in = line && y >= 0 && y < H;
                    copy16_async(rg + c, in ? bloom + at + c : bloom, in ? 16 : 0);
                    copy8_async(b + c, in ? bl + at + c : bl, in ? 8 : 0);
                }
            }
            at += (ptrdiff_t)kTWarps * H;
            rg += kTWarps * stride;
            b += kTWarps * stride;
        }
    } else {
        const int p = tid & (kTPairs - 1), x = x0 + 2 * p;
#pragma unroll 4
        for (int c = tid / kTPairs; c < segw; c += kTThreads / kTPairs) {
            const int y = y0 - R + c;
            const bool in = y >= 0 && y < H;
            const float4* row = bloom + (size_t)(in ? y : 0) * W;
            float4 u = make_float4(0.f, 0.f, 0.f, 0.f), v = u;
            if (in && x < W) u = load_behind_wait(row + x);
            if (in && x + 1 < W) v = load_behind_wait(row + x + 1);
            t.rg[p * stride + c] = make_ulonglong2(pack2(u.x, v.x), pack2(u.y, v.y));
            t.b[p * stride + c] = pack2(u.z, v.z);
        }
    }
    copy_async_wait_all();
    __syncthreads();
    const int p = tid & (kTPairs - 1), cb = (tid / kTPairs) * kBJ;
    const int x = x0 + 2 * p, ys = y0 + cb;
    if (x >= W || ys >= H) return;
    const bool second = x + 1 < W;
    uint64_t acc[kBJ][3];
    blur_pair(t.rg + p * stride + cb, t.b + p * stride + cb, t.w, R, acc);
    // composite sources 4 rows ahead of their tone maps
    constexpr int kAhead = 4;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 us[kAhead], vs[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
        const float4* at = hdr + (size_t)(ys + j) * W + x;
        us[j] = ys + j < H ? load_behind_wait(at) : zero;
        vs[j] = ys + j < H && second ? load_behind_wait(at + 1) : zero;
    }
#pragma unroll
    for (int j = 0; j < kBJ; ++j) {
        const int y = ys + j;
        if (y >= H) break;
        const size_t idx = (size_t)y * W + x;
        const float s = t.inv[cb + j];
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[j][c] = mul2(acc[j][c], pack2(s, s));
        const float4 u = us[j % kAhead], v = vs[j % kAhead];
        if (j + kAhead < kBJ) {
            const float4* at = hdr + (size_t)(y + kAhead) * W + x;
            us[j % kAhead] = y + kAhead < H ? load_behind_wait(at) : zero;
            vs[j % kAhead] = y + kAhead < H && second ? load_behind_wait(at + 1) : zero;
        }
        image[idx] = tone_pack(u.x + lo2(acc[j][0]) * pp.intensity, u.y + lo2(acc[j][1]) * pp.intensity,
                               u.z + lo2(acc[j][2]) * pp.intensity);
        if (second)
            image[idx + 1] = tone_pack(v.x + hi2(acc[j][0]) * pp.intensity, v.y + hi2(acc[j][1]) * pp.intensity,
                                       v.z + hi2(acc[j][2]) * pp.intensity);
    }
}

// The same from a row-major bloom buffer for radii whose tile does not fit in shared memory: one
// pixel per thread, the reference's loop.
__global__ void __launch_bounds__(256) post_v_wide_kernel(const PostParams pp, const float4* __restrict__ hdr,
                                                          const float4* __restrict__ bloom,
                                                          uint32_t* __restrict__ image) {
    const int x = blockIdx.x * 32 + (threadIdx.x & 31), y = blockIdx.y * 8 + (threadIdx.x >> 5);
    if (x >= pp.width || y >= pp.height) return;
    const int R = pp.radius;
    float ax = 0.0f, ay = 0.0f, az = 0.0f;
    for (int i = max(-R, -y); i <= min(R, pp.height - 1 - y); ++i) {
        const float w = __ldg(&pp.weights[i + R].x);
        const float4 c = __ldg(bloom + (size_t)(y + i) * pp.width + x);
        ax += c.x * w;
        ay += c.y * w;
        az += c.z * w;
    }
    const float s = __ldg(pp.inv_wsum_y + y);
    const size_t idx = (size_t)y * pp.width + x;
    const float4 base = __ldg(hdr + idx);
    image[idx] = tone_pack(base.x + __fmul_rn(ax, s) * pp.intensity, base.y + __fmul_rn(ay, s) * pp.intensity,
                           base.z + __fmul_rn(az, s) * pp.intensity);
}

// Tone map only (bloom inactive): 4 pixels per thread, their loads issued together.
__global__ void __launch_bounds__(256) tonemap_kernel(const PostParams pp, const float4* __restrict__ hdr,
                                                      uint32_t* __restrict__ image) {
    const size_t n = (size_t)pp.width * pp.height;
    const size_t i0 = (size_t)blockIdx.x * 1024 + threadIdx.x;
    float4 c[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) c[k] = i0 + 256 * k < n ? __ldg(hdr + i0 + 256 * k) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (i0 + 256 * k < n) image[i0 + 256 * k] = tone_pack(c[k].x, c[k].y, c[k].z);
}

// The blur's tables, made once per context: weight pairs 0 .. 2R (and a zero behind them), and for every
// column and row the reciprocal of the sum of its in-image weights, added in tap order (1 where the
// sum is 0).
__global__ void __launch_bounds__(256) post_weights_kernel(int R, float sigma, float2* __restrict__ weights) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const float w = i <= 2 * R ? tap_weight(i - R, sigma) : 0.0f;
    if (i <= 2 * R + 1) weights[i] = make_float2(w, w);
}
__global__ void __launch_bounds__(256) post_weight_sums_kernel(const PostParams pp, float* __restrict__ inv_x,
                                                               float* __restrict__ inv_y) {
    const int R = pp.radius;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int axis = i < pp.width ? 0 : 1, pos = axis ? i - pp.width : i, n = axis ? pp.height : pp.width;
    if (i >= pp.width + pp.height) return;
    float ws = 0.0f;
    for (int k = max(-R, -pos); k <= min(R, n - 1 - pos); ++k) ws += pp.weights[k + R].x;
    (axis ? inv_y : inv_x)[pos] = ws > 0.0f ? 1.0f / ws : 1.0f;
}

constexpr size_t kSmemLimit = 200 * 1024;
// Largest radius of the horizontal pass and the fused post.  The tiles of line pairs would take radii up to
// 229 in kSmemLimit; this is the limit that callers know, at which tiles of 32 single lines filled it, and
// a radius that was refused stays refused.  The vertical pass alone has no such limit: it takes the
// tiles as far as they go and post_v_wide_kernel beyond.
constexpr int kMaxRadius = 165;
static_assert(pair_smem(kMaxRadius) <= kSmemLimit, "the largest radius fits its tile");
static bool radius_fits(int R) { return R <= kMaxRadius; }

// Lets a kernel be launched with `bytes` of shared memory.  The attribute belongs to the function, not
// to the launch, so it is always raised to the same limit: with the size of the call at hand, a
// thread with a smaller radius could lower it between another's call and launch, which then failed.
static cudaError_t set_smem(const void* fn, size_t bytes) {
    if (bytes <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit);
}

// Radii above this (25583) are refused by every post entry point and have no tables.
static bool radius_has_tables(int R) { return ((size_t)2 * R + 2 + 32) * sizeof(float) <= kSmemLimit; }

size_t post_table_floats(const PostParams& pp) {
    return radius_has_tables(pp.radius) ? 2 * ((size_t)2 * pp.radius + 2) + pp.width + pp.height : 0;
}

cudaError_t launch_post_tables(PostParams& pp, float* tables, cudaStream_t st) {
    if (!radius_has_tables(pp.radius)) return cudaSuccess;
    const int nw = 2 * pp.radius + 2;
    float2* weights = reinterpret_cast<float2*>(tables);
    float* sums = tables + 2 * (size_t)nw;
    pp.weights = weights;
    pp.inv_wsum_x = sums;
    pp.inv_wsum_y = sums + pp.width;
    post_weights_kernel<<<(nw + 255) / 256, 256, 0, st>>>(pp.radius, pp.sigma, weights);
    post_weight_sums_kernel<<<(pp.width + pp.height + 255) / 256, 256, 0, st>>>(pp, sums, sums + pp.width);
    return cudaGetLastError();
}

static cudaError_t launch_tonemap(const PostParams& pp, const float4* hdr, uint32_t* image, cudaStream_t st) {
    const size_t n = (size_t)pp.width * pp.height;
    tonemap_kernel<<<(unsigned)((n + 1023) / 1024), 256, 0, st>>>(pp, hdr, image);
    return cudaGetLastError();
}

template <bool PAIRED>
static cudaError_t launch_h(const PostParams& pp, const float4* hdr, float4* bloom, cudaStream_t st) {
    // the row-major output's transposition takes kTPairs x (kTPos + 1) float4 of the staged tile
    const size_t sm = std::max(pair_smem(pp.radius), (size_t)kTPairs * (kTPos + 1) * 16);
    const cudaError_t e = set_smem((const void*)bloom_h_kernel<PAIRED>, sm);
    if (e != cudaSuccess) return e;
    const dim3 grid((pp.width + kTPos - 1) / kTPos, (pp.height + 2 * kTPairs - 1) / (2 * kTPairs));
    return launch_early(bloom_h_kernel<PAIRED>, grid, kTThreads, sm, st, pp, hdr, bloom);
}
template <bool PAIRED>
static cudaError_t launch_v(const PostParams& pp, const float4* hdr, const float4* bloom, uint32_t* image,
                            cudaStream_t st) {
    const size_t sm = pair_smem(pp.radius);
    const cudaError_t e = set_smem((const void*)post_v_kernel<PAIRED>, sm);
    if (e != cudaSuccess) return e;
    const dim3 grid((pp.width + 2 * kTPairs - 1) / (2 * kTPairs), (pp.height + kTPos - 1) / kTPos);
    return launch_early(post_v_kernel<PAIRED>, grid, kTThreads, sm, st, pp, hdr, bloom, image);
}

cudaError_t launch_bloom_horizontal(const PostParams& pp, const float4* hdr, float4* bloom, cudaStream_t st) {
    if (pp.width <= 0 || pp.height <= 0) return cudaSuccess;
    if (!radius_fits(pp.radius)) return cudaErrorInvalidValue;
    return launch_h<false>(pp, hdr, bloom, st);
}

cudaError_t launch_post_process(const PostParams& pp, const float4* hdr, const float4* bloom,
                                uint32_t* image, cudaStream_t st) {
    if (pp.width <= 0 || pp.height <= 0) return cudaSuccess;
    if (!pp.active) return launch_tonemap(pp, hdr, image, st);
    if (pair_smem(pp.radius) <= kSmemLimit) return launch_v<false>(pp, hdr, bloom, image, st);
    if (!radius_has_tables(pp.radius)) return cudaErrorInvalidValue;
    const dim3 grid((pp.width + 31) / 32, (pp.height + 7) / 8);
    post_v_wide_kernel<<<grid, 256, 0, st>>>(pp, hdr, bloom, image);
    return cudaGetLastError();
}

cudaError_t launch_post_fused(const PostParams& pp, const float4* hdr, uint32_t* image, float4* scratch,
                              cudaStream_t st) {
    if (pp.width <= 0 || pp.height <= 0) return cudaSuccess;
    if (!pp.active) return launch_tonemap(pp, hdr, image, st);
    if (!scratch || !radius_fits(pp.radius)) return cudaErrorInvalidValue;
    const cudaError_t e = launch_h<true>(pp, hdr, scratch, st);
    return e != cudaSuccess ? e : launch_v<true>(pp, hdr, scratch, image, st);
}

// FP32 FMA throughput probe (the denominator of the trace's roofline): eight independent
// dependent chains per thread hide the FMA latency; the chains are kept alive by a store that
// only a sum of exactly 12345.678 would trigger.
__global__ void __launch_bounds__(512) fma_probe_kernel(float b, float c, int iters, float* sink) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = (float)threadIdx.x * 1e-3f + (float)i;
#pragma unroll 8
    for (int k = 0; k < iters; ++k) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = fmaf(v[i], b, c);
    }
    float s = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += v[i];
    if (s == 12345.678f) sink[0] = s;
}

cudaError_t launch_fma_probe(int blocks, int iters, float* sink, cudaStream_t st) {
    fma_probe_kernel<<<blocks, 512, 0, st>>>(0.999999f, 1e-6f, iters, sink);
    return cudaGetLastError();
}

}  // namespace ktd
