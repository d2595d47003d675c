// kt_internal.h — launchers shared by the C-ABI layer (kt_host.cpp) and the kernels
// translation unit (kt_kernels.cu).  Not part of the public ABI.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "kt_types.h"

namespace ktd {

// Bloom / post-process constants of one context (src/renderer/init.rs:43-73, mod.rs:139-148).
struct PostParams {
    int width, height;
    int radius;       // ceil(bloom.radius)
    float sigma;      // bloom.radius / 3
    float intensity;
    int active;       // enabled && radius > 0 && intensity > 0
    int mode;         // stated-physics luminance threshold when 1
    float threshold;
    // device tables of the blur (launch_post_tables; also when bloom is inactive, for the separate passes)
    const float2* weights;    // 2 radius + 1 tap weights, each twice, and a zero
    const float* inv_wsum_x;  // per column, per row: 1 / the sum of the in-image weights
    const float* inv_wsum_y;
};

// Tuning of the persistent tracer: resident blocks per SM (3..6 for the FP32 reference
// kernel; the default otherwise).  refill_min is carried for its callers and has no effect.
struct Tuning {
    int schedule = 1;
    int block_x = 0, block_y = 0;
    int blocks_per_sm = 4;
    int refill_min = 1;
    int order = 0;  // 1: pixels ranked long-rays-first by the rank kernel before the trace
    int keep_frozen = 0;  // 1: NaN-frozen rays iterate to max_steps (Scene::keep_frozen)
};

// Pixel-order buffer: kOrderHeader header words (marked / unmarked counts), then one pixel
// index per work unit.
constexpr unsigned kOrderHeader = 16;

// Trace launch: schedule 0 = plain 2D grid (block bx x by), 1 = persistent wavefront.
// precision 0 = FP32, 1 = mixed, 2 = FP64.  queue: one device word, reset here on `stream`.
// ctr: optional 6 x u64 device counters (selects the counting kernels); aux: optional float4
// per pixel with the first shaded disk hit (r, g, T, hits) of sample 0 (counting kernels only).
// order: NULL for tile order, else a pixel-order buffer of kOrderHeader + width * height words
// that the rank kernel fills on `stream` before the trace.
cudaError_t launch_trace(const Scene& sc, const Camera& cam, int schedule, float4* hdr,
                         uint32_t* err, unsigned* queue, unsigned long long* ctr, float4* aux,
                         const Tuning& tn, int bx, int by, unsigned* order, cudaStream_t stream);

// ---- order in which the units take the pixels of a frame ---------------------------------------
// A unit is a run of 32 / S indices; frame_pixel turns an index into a pixel.  Patches: 16x16 tiles in
// raster order, Morton order inside a tile, so that an aligned run of 32, 16, 8, ... indices is a
// patch of 8x4, 4x4, 4x2, ... pixels.  The indices cover whole tiles: some name no pixel.  Strips: the
// frame cut into strips of about 8 columns, each numbered row by row, one after the other: exactly
// one index per pixel, and a run of 32 is about as square.
//
// In frames with short sides the patches leave lanes idle: 28 of 32 at one column, 24 at one row, a
// third at 17 columns.  A launch that fills the GPU pays for them, so it takes strips where less than
// 15 of 16 lanes of the patches with a pixel have one (below about 110 columns or 60 rows).
// Patches -> strips, FP32: 64 persistent renders of 1x8192 5.42 -> 0.77 ms, of 17x4096 8.17 -> 5.74; a
// frame of 1x32768 374 -> 103 us; eight views of it 2.64 -> 0.41 ms; recording forward of 9x32768 609 ->
// 388 us.
// A launch whose patches all start at once lasts as long as its longest warp, and a warp with idle
// lanes is shorter: it keeps the patches.
// (patches and strips: frame of 1x1080 80 and 97 us, recording forward in FP64 of 300x33 334 and 385.)
// The kernels are instances for one order or the other: with both in one, the large launches of the
// mixed trace and of the views call were 0.5% slower.  Launch shapes of the wavefront schedule other
// than the default (blocks per SM, counting) keep the patches.
__host__ __device__ inline bool patches_idle(int W, int H) {
    const unsigned w = ((unsigned)W + 7u) & ~7u, h = ((unsigned)H + 3u) & ~3u;
    return 16ull * ((unsigned)W * (unsigned)H) < 15ull * (w * h);
}
// Indices of a frame.
__host__ __device__ inline unsigned index_count(int W, int H, bool strips) {
    return strips ? (unsigned)W * (unsigned)H : ((unsigned)(W + 15) >> 4) * ((unsigned)(H + 15) >> 4) * 256u;
}
// The pixel of an index; false when it has none (outside the frame, or beyond the last index).
__host__ __device__ inline bool frame_pixel(unsigned idx, int W, int H, bool strips, int& px, int& py) {
    if (strips) {
        // n strips, strip i from column i W / n on: i W / n H indices lie before it, so idx / H is one
        // of the columns of idx's strip
        const unsigned n = W < 12 ? 1u : ((unsigned)W + 4u) >> 3;
        const unsigned column = idx / (unsigned)H;
        const unsigned strip = ((column + 1u) * n - 1u) / (unsigned)W;
        const unsigned x0 = strip * (unsigned)W / n, x1 = (strip + 1u) * (unsigned)W / n;
        const unsigned at = idx - x0 * (unsigned)H, w = x1 - x0;
        py = (int)(at / w);
        px = (int)(x0 + at - (unsigned)py * w);
        return column < (unsigned)W;
    }
    const unsigned tiles_x = ((unsigned)W + 15u) >> 4;
    const unsigned tile = idx >> 8, m = idx & 255u;
    const unsigned ty = tile / tiles_x, tx = tile - ty * tiles_x;
    const unsigned x = (m & 1u) | (m >> 1 & 2u) | (m >> 2 & 4u) | (m >> 3 & 8u);
    const unsigned y = (m >> 1 & 1u) | (m >> 2 & 2u) | (m >> 3 & 4u) | (m >> 4 & 8u);
    px = (int)(tx * 16u + x);
    py = (int)(ty * 16u + y);
    return px < W && py < H;
}
// Units of 32 / S pixels that cover a frame: all its indices, or exactly its pixels when they come
// from a pixel-order buffer.
__host__ __device__ inline unsigned unit_count(int W, int H, int S, bool ordered, bool strips) {
    const unsigned P = 32u / (unsigned)S;
    const unsigned n = ordered ? (unsigned)W * (unsigned)H : index_count(W, H, strips);
    return (n + P - 1u) / P;
}
// The rule above: whether a frame takes strips in a launch of `patch_units` units, counted in patches
// over all its frames, on a GPU that holds `warps` of the kernel's warps.
inline bool take_strips(int W, int H, unsigned patch_units, unsigned warps) {
    return patch_units > warps && patches_idle(W, H);
}

#ifdef __CUDACC__
// A launch that may start before the stream's previous kernel has ended: its blocks come up, and do what
// touches no memory that another kernel writes or reads (tables made with the context may be read),
// while that one drains, and call wait_for_stream() before the rest.  wait_for_stream() returns
// when everything ahead in the stream has ended and its writes are visible, so every kernel launched
// this way keeps the stream's order; it does nothing in a kernel launched the plain way.  What it
// saves is the gap between two launches, about 2 us each (back to back, launched the plain way and this
// way): fused post of 96x64 15.4 -> 11.5 us, 960x540 20.5 -> 16.1, 1920x1080 45.1 -> 41.1, 3840x2160
// 162.9 -> 159.2 (two launches); the two tables of 4096 rows 11.3 -> 7.1 (two); a 96x64 frame of 2
// samples with its post 117.7 -> 110 (three).
template <class F, class... A>
cudaError_t launch_early(F kernel, dim3 grid, int block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}
__device__ __forceinline__ void wait_for_stream() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// A load of what an earlier kernel of the stream wrote.  A const __restrict__ pointer or __ldg makes a
// load that the compiler may move ahead of the wait; this one stays behind it.
__device__ __forceinline__ float4 load_behind_wait(const float4* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
// Lets the next launch_early kernel of the stream come up as soon as every block has called this or ended.
__device__ __forceinline__ void let_next_launch() { asm volatile("griddepcontrol.launch_dependents;"); }
#endif

// Batched trace: one plain-schedule launch over the tiles of up to kBatchMaxJobs renders.  The
// table travels as a kernel parameter (__grid_constant__); each block finds its job from the
// tile prefix, so the job index and its scene constants are uniform across the block.
constexpr int kBatchMaxJobs = 64;
struct BatchJob {
    Scene sc;
    Camera cam;
    float4* hdr;
    uint32_t* err;
    int tiles_x;
    int tile_begin;
    unsigned unit_begin;  // persistent launch: first 32-pixel unit of this job
    int strips;           // and its pixel order
};
struct BatchTable {
    BatchJob job[kBatchMaxJobs];
    int n;
    int total_tiles;
    unsigned total_units;
};
cudaError_t launch_batch(const BatchTable& bt, int bx, int by, cudaStream_t stream);
// Persistent batched trace: warps take 32-pixel units, each inside one job, from the device
// counter `counter` (one word, reset here on `stream` when it is used); blocks of 128 threads, blocks_per_sm
// resident per SM (the FP32 reference-semantics kernel has 4, 5 and 6; the others their default).
cudaError_t launch_batch_persistent(const BatchTable& bt, int blocks_per_sm, unsigned* counter, cudaStream_t stream);
// Number of 16-byte words that differ between a and b (n16 words each) into *out (device).
cudaError_t launch_count_mismatch(const void* a, const void* b, size_t n16, unsigned long long* out,
                                  cudaStream_t stream);

cudaError_t launch_bloom_horizontal(const PostParams& pp, const float4* hdr, float4* bloom,
                                    cudaStream_t stream);
cudaError_t launch_post_process(const PostParams& pp, const float4* hdr, const float4* bloom,
                                uint32_t* image, cudaStream_t stream);
// Fills pp's tables (post_table_floats(pp) floats of device memory at `tables`) on `stream`.
size_t post_table_floats(const PostParams& pp);
cudaError_t launch_post_tables(PostParams& pp, float* tables, cudaStream_t stream);
// Both post passes; scratch: post_scratch_bytes(width, height) of device memory for the bloom buffer
// (unused when bloom is off).
size_t post_scratch_bytes(int width, int height);
cudaError_t launch_post_fused(const PostParams& pp, const float4* hdr, uint32_t* image, float4* scratch,
                              cudaStream_t stream);
// FP32 FMA throughput probe: `blocks` x 512 threads, each running 8 independent FMA chains of
// `iters` steps (16 * iters flops per thread).
cudaError_t launch_fma_probe(int blocks, int iters, float* sink, cudaStream_t st);
// Lookup tables on the device (kt_luts.cu): n_lambda wavelengths from wl_start in steps of
// wl_step; disk radii from r_in to r_out.
cudaError_t launch_blackbody_lut(uint32_t size, float max_temp, float wl_start, int n_lambda, float wl_step,
                                 float4* out, cudaStream_t st);
cudaError_t launch_disk_lut(uint32_t size, float a_norm, float inv_m, float r_in, float r_out, float* out,
                            cudaStream_t st);

}  // namespace ktd

// Host helpers shared with the allocation-free entry point (kt_noalloc.cu).
#include "../../include/kerrtrace.h"
namespace ktd {
kt_status scene_from_config(const kt_config* cfg, Scene* out);
kt_status set_error(kt_status s, const char* msg);
}  // namespace ktd
