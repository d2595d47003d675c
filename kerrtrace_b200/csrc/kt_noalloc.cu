// kt_noalloc.cu — trace entry point that allocates no device memory (kt_trace_noalloc).
//
// Some callers cannot allocate device memory at the point where they render: a host whose
// device memory all belongs to its own pool allocator (an engine, or a framework with a caching
// allocator that must account for every byte), or a per-frame path that must not call
// cudaMalloc / cudaFree because they synchronise the device and would stall the frames already
// in flight.  Such a caller cannot create a kt_context, which allocates its LUT textures and
// its work counter.  kt_trace_noalloc takes everything from the caller instead — scene
// configuration, cameras, the two LUTs as plain device arrays, the output buffers — and keeps
// its only scratch, a work counter, in the file-scope word below.
//
// The word is part of the library's device image: every GPU that loads the library holds it
// until the process exits.  Every call shares it and it keeps the last call's
// count; a call that uses it clears it on its own stream before the trace kernel runs.  Calls that
// overlap on the GPU (other streams, other host threads on the same device) race on it and must
// be serialised by the caller.
//
// The kernel is the persistent tracer with reference semantics; the LUTs are read
// from the plain arrays through a model of the texture unit's linear filter (mode 2 of the
// device code), so results agree with kt_trace to the parity tolerance, not bit for bit.
#include <cuda_runtime.h>

#include <cstdio>
#include <mutex>

#include "../../include/kerrtrace.h"
#include "kt_internal.h"
#include "kt_ray.cuh"

namespace ktd {

// Scratch of kt_trace_noalloc: the work counter, on a 128-byte line of its own.  In host code this name is
// only a stand-in for the device symbol; its device address comes from cudaGetSymbolAddress.
static __device__ __align__(128) unsigned int g_noalloc_queue;

struct NoallocViews {
    Camera cam[KT_NOALLOC_MAX_VIEWS];
    int n;
};

constexpr unsigned kFullMask = 0xffffffffu;
constexpr int kNoallocBlock = 128;

// Persistent trace over several views of one scene, in the units of trace_wavefront_kernel: 32 / S
// pixels with S samples of each side by side, view after view.  A warp's first unit is its own index
// in the grid, the others come from one counter over all views.  (Refilling single lanes, as an
// earlier form did, ran the ray set-up for one lane of 32: 8 views of 480x270 1.78 ms, now 1.22; at
// 4 samples 8.55, now 4.59; 12 views of 64x36 at 2 samples 418 us, now 162.)
template <bool TOGETHER, bool STRIPS>
__global__ void __launch_bounds__(kNoallocBlock, 4)
    trace_views_noalloc_kernel(const __grid_constant__ Scene sc, const __grid_constant__ NoallocViews views,
                               float4* __restrict__ hdr, uint32_t* __restrict__ err, unsigned* __restrict__ queue,
                               int S) {
    constexpr int MODE = 2;
    const int lane = threadIdx.x & 31;
    const int slot = lane / S, sub = lane - slot * S;
    const unsigned P = 32u / (unsigned)S;
    const unsigned per_view = unit_count(sc.width, sc.height, S, false, STRIPS);
    const unsigned units = per_view * (unsigned)views.n;
    const unsigned n_warps = gridDim.x * (kNoallocBlock / 32);
    const size_t n_px = (size_t)sc.width * sc.height;
    for (unsigned u = blockIdx.x * (kNoallocBlock / 32) + (threadIdx.x >> 5); u < units;) {
        const unsigned view = u / per_view;
        const Camera& cam = views.cam[view];
        int px = 0, py = 0;
        const bool valid = (unsigned)slot < P && frame_pixel((u - view * per_view) * P + (unsigned)slot, sc.width,
                                                             sc.height, STRIPS, px, py);
        float acc[3] = {0.0f, 0.0f, 0.0f};
        for (int s0 = 0; s0 < sc.spp; s0 += S) {
            const int smp = s0 + sub;
            RayRun<float> ry;
            Tally tl;
            bool run = false;
            float col[3] = {0.0f, 0.0f, 0.0f};
            if (valid && smp < sc.spp) {
                float dir[3];
                pixel_ray<MODE>(px, py, smp, sc, cam, dir);
                run = ray_start<float>(ry, cam, dir, sc, smp > 0);
            }
            run_rays<MODE, false, TOGETHER>(run, ry, sc, err + 2 * view, tl);
            if (run) {
#pragma unroll
                for (int c = 0; c < 3; ++c) col[c] = ry.col[c];
            }
            const int last = min(S, sc.spp - s0);
            for (int i = 0; i < last; ++i) {
#pragma unroll
                for (int c = 0; c < 3; ++c) acc[c] += __shfl_sync(kFullMask, col[c], min(slot * S + i, 31));
            }
        }
        if (valid && sub == 0) {
            const float fs = sc.final_scale;
            hdr[view * n_px + (size_t)py * sc.width + px] = make_float4(acc[0] * fs, acc[1] * fs, acc[2] * fs, 1.0f);
        }
        if (units <= n_warps) break;
        if (lane == 0) u = n_warps + atomicAdd(queue, 1u);
        u = __shfl_sync(kFullMask, u, 0);
    }
}

// Device address of g_noalloc_queue, looked up once per device.
constexpr int kMaxDevices = 64;
static std::mutex g_noalloc_mutex;
static unsigned* g_noalloc_addr[kMaxDevices];

static kt_status noalloc_scratch(int device, unsigned** out) {
    if (device < 0 || device >= kMaxDevices) return set_error(KT_ERR_INVALID_ARG, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_addr[device]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_queue);
        if (e != cudaSuccess) {
            char msg[256];
            snprintf(msg, sizeof msg, "cudaGetSymbolAddress of the work counter failed: %s", cudaGetErrorString(e));
            return set_error(KT_ERR_CUDA, msg);
        }
        g_noalloc_addr[device] = static_cast<unsigned*>(p);
    }
    *out = g_noalloc_addr[device];
    return KT_OK;
}

}  // namespace ktd

extern "C" kt_status kt_trace_noalloc(const kt_config* cfg, const kt_camera* cams, uint32_t n_views,
                                      const float* bb_lut, const float* disk_lut, void* stream,
                                      float* hdr_out, uint32_t* err_words) {
    using namespace ktd;
    if (!cfg || !cams || !bb_lut || !disk_lut || !hdr_out || !err_words)
        return set_error(KT_ERR_INVALID_ARG, "kt_trace_noalloc: NULL argument");
    if (n_views == 0 || n_views > KT_NOALLOC_MAX_VIEWS) {
        char msg[160];
        snprintf(msg, sizeof msg, "kt_trace_noalloc: %u views requested; its table of cameras holds 1..%d",
                 n_views, KT_NOALLOC_MAX_VIEWS);
        return set_error(KT_ERR_INVALID_ARG, msg);
    }
    if (cfg->mode != KT_MODE_REF || cfg->precision != KT_PREC_FP32)
        return set_error(KT_ERR_UNSUPPORTED, "kt_trace_noalloc implements the reference semantics in FP32 only");
    if ((uint64_t)cfg->width * cfg->height * n_views >= (1ull << 32))
        return set_error(KT_ERR_INVALID_ARG, "kt_trace_noalloc: frame too large for the 32-bit work counter");
    Scene sc;
    kt_status st = scene_from_config(cfg, &sc);
    if (st != KT_OK) return st;
    sc.bb_lut = reinterpret_cast<const float4*>(bb_lut);
    sc.disk_lut = disk_lut;
    sc.bb_tex = 0;
    sc.disk_tex = 0;
    NoallocViews views;
    views.n = (int)n_views;
    for (uint32_t v = 0; v < n_views; ++v) {
        for (int i = 0; i < 3; ++i) {
            views.cam[v].pos[i] = cams[v].cam_pos[i];
            views.cam[v].fwd[i] = cams[v].fwd[i];
            views.cam[v].rgt[i] = cams[v].rgt[i];
            views.cam[v].up[i] = cams[v].up[i];
        }
        views.cam[v].fov_scale = cams[v].fov_scale;
    }
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_error(KT_ERR_CUDA, "cudaGetDevice failed");
    unsigned* queue = nullptr;
    if ((st = noalloc_scratch(dev, &queue)) != KT_OK) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
        return set_error(KT_ERR_CUDA, cudaGetErrorString(e));
    constexpr unsigned kWarps = kNoallocBlock / 32;
    int S = samples_in_parallel(sc.spp);
    // the unit counter is 32 bits wide (whole tiles of a large frame, up to a unit per pixel)
    if ((uint64_t)unit_count(sc.width, sc.height, S, false, false) * n_views > 0x7fffffffu) S = 1;
    const unsigned resident = (unsigned)sms * 4u;
    const bool strips = take_strips(sc.width, sc.height, unit_count(sc.width, sc.height, S, false, false) * n_views,
                                    resident * kWarps);
    const unsigned units = unit_count(sc.width, sc.height, S, false, strips) * n_views;
    const unsigned blocks = (units + kWarps - 1) / kWarps;
    const unsigned grid = blocks < resident ? blocks : resident;
    float4* hdr = reinterpret_cast<float4*>(hdr_out);
    if (units <= grid * kWarps && !strips) {  // one unit per warp: lanes in step, as in launch_wave_minb
        trace_views_noalloc_kernel<true, false><<<grid, kNoallocBlock, 0, s>>>(sc, views, hdr, err_words, queue, S);
    } else {
        if ((e = cudaMemsetAsync(queue, 0, sizeof(unsigned), s)) != cudaSuccess)
            return set_error(KT_ERR_CUDA, cudaGetErrorString(e));
        if (strips)
            trace_views_noalloc_kernel<false, true><<<grid, kNoallocBlock, 0, s>>>(sc, views, hdr, err_words, queue, S);
        else
            trace_views_noalloc_kernel<false, false><<<grid, kNoallocBlock, 0, s>>>(sc, views, hdr, err_words, queue, S);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return set_error(KT_ERR_CUDA, cudaGetErrorString(e));
    return KT_OK;
}
