// kt_host.cpp — C-ABI layer: host precompute, device context, CudaRenderer mirror.
//
// Host precompute restates the reference's Rust host in f32 arithmetic with the same libm
// calls (Rust's f32::{cbrt, acos, cos, ln, exp, exp_m1} are the C library's cbrtf, acosf, cosf,
// logf, expf, expm1f; mul_add is fmaf; this file is built with -ffp-contract=off so that no
// other product is fused):
//   build_kerr_params            src/renderer/utils.rs:53-113
//   calc_isco                    src/renderer/utils.rs:11-20
//   calc_novikov_thorne_factor   src/renderer/utils.rs:21-52
//   generate_disk_temperature_lut src/renderer/utils.rs:172-201
//   generate_blackbody_lut       src/renderer/blackbody.rs:6-124
//   build_cuda_defines           src/renderer/utils.rs:115-163
//   validate_bloom_settings      src/renderer/init.rs:43-73
//   f32_from_f64                 src/math.rs:15-32 (shortest round-trip text, then parse)
// Device context and renderer follow src/renderer/{texture,init,mod}.rs.
#include <cuda_runtime.h>

#include <algorithm>
#include <charconv>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <limits>
#include <new>
#include <string>
#include <vector>

#include "../../include/kerrtrace.h"
#include "kt_context.h"
#include "kt_internal.h"

namespace {

thread_local std::string g_last_error;

kt_status fail(kt_status s, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_last_error = buf;
    return s;
}
kt_status cuda_fail(cudaError_t e, const char* what) {
    return fail(KT_ERR_CUDA, "%s: %s (%s)", what, cudaGetErrorName(e), cudaGetErrorString(e));
}
#define KT_CUDA(call, what)                              \
    do {                                                 \
        cudaError_t e__ = (call);                        \
        if (e__ != cudaSuccess) return cuda_fail(e__, what); \
    } while (0)

// ---- numeric helpers ---------------------------------------------------------------------

// src/math.rs:15-32: the f64 is printed with its shortest round-trip digits and that text is
// parsed as f32.  The text's value lies within half an ulp of the f64, so it rounds to the same f32
// as the f64 itself unless the midpoint of two f32 is that close: only then (and for subnormal
// results) the text is made (about 150 ns against 2; the tables convert every entry).
bool f32_from_f64(double v, float* out) {
    if (!std::isfinite(v)) return false;
    if (v < -(double)std::numeric_limits<float>::max() || v > (double)std::numeric_limits<float>::max()) return false;
    uint64_t bits;
    std::memcpy(&bits, &v, sizeof bits);
    const uint32_t below = (uint32_t)(bits & 0x1fffffffu);  // the 29 bits that f32 does not keep
    if ((below < 0x0fffffffu || below > 0x10000001u) && std::fabs(v) >= (double)std::numeric_limits<float>::min()) {
        const float f = (float)v;
        if (!std::isfinite(f)) return false;
        *out = f;
        return true;
    }
    char buf[64];
    auto res = std::to_chars(buf, buf + sizeof buf - 1, v);
    if (res.ec != std::errc()) return false;
    *res.ptr = '\0';
    const float f = std::strtof(buf, nullptr);
    if (!std::isfinite(f)) return false;
    *out = f;
    return true;
}

// Value of the reference's `#define KEY {value:.10}` as the double literal the compiler sees.
double define_value(float v) {
    char buf[128];
    snprintf(buf, sizeof buf, "%.10f", (double)v);
    return std::strtod(buf, nullptr);
}
float float_ceil(double d) {  // smallest float >= d
    float f = (float)d;
    if ((double)f < d) f = std::nextafterf(f, std::numeric_limits<float>::infinity());
    return f;
}
float float_floor(double d) {  // largest float <= d
    float f = (float)d;
    if ((double)f > d) f = std::nextafterf(f, -std::numeric_limits<float>::infinity());
    return f;
}

float isco_f32(float a_norm, bool prograde, float mass) {
    const float aa = a_norm * a_norm;
    const float z1 = fmaf(cbrtf(1.0f - aa), cbrtf(1.0f + a_norm) + cbrtf(1.0f - a_norm), 1.0f);
    const float z2 = sqrtf(fmaf(3.0f, aa, z1 * z1));
    const float sign = prograde ? -1.0f : 1.0f;
    const float inside = (3.0f - z1) * fmaf(2.0f, z2, 3.0f + z1);
    return mass * (3.0f + z2 + sign * sqrtf(fmaxf(inside, 0.0f)));
}

// Page-Thorne flux factor with the roots 2 cos(acos(-a)/3 - 2 pi k / 3) of x^3 - 3x + 2a = 0.  What
// depends on the spin and the ISCO alone is computed once per table.
struct NtTerms {
    float roots[3], den[3], coef[3], x_ms;
};
NtTerms nt_terms_f32(float a_norm, float r_isco, float inv_m) {
    NtTerms t;
    t.x_ms = sqrtf(r_isco * inv_m);
    const float third = 1.0f / 3.0f;
    const float angle_base = acosf(-a_norm) * third;
    const float ang_step = 2.0943952f;
    t.roots[0] = 2.0f * cosf(angle_base);
    t.roots[1] = 2.0f * cosf(angle_base - ang_step);
    t.roots[2] = 2.0f * cosf(angle_base + ang_step);
    for (int i = 0; i < 3; ++i) {
        const float xi = t.roots[i];
        t.den[i] = xi * (xi - t.roots[(i + 1) % 3]) * (xi - t.roots[(i + 2) % 3]);
        t.coef[i] = 3.0f * (xi - a_norm) * (xi - a_norm) / t.den[i];
    }
    return t;
}
float nt_factor_f32(float r, float a_norm, float r_isco, float inv_m, const NtTerms& t) {
    if (r <= r_isco) return 0.0f;
    const float r_norm = r * inv_m;
    const float x = sqrtf(r_norm);
    const float x_ms = t.x_ms;
    float sum_log = 0.0f;
    for (int i = 0; i < 3; ++i) {
        if (t.den[i] <= 0.0f) continue;
        const float val = (x - t.roots[i]) / (x_ms - t.roots[i]);
        if (val > 0.0f) sum_log += t.coef[i] * logf(val);
    }
    const float q = fmaf(1.5f * a_norm, -logf(x / x_ms), x - x_ms) - sum_log;
    const float geo = r_norm * fmaf(2.0f, a_norm, fmaf(r_norm, x, -(3.0f * x)));
    return fmaxf(q / geo, 0.0f);
}

float cmf_lobe(float x, float alpha, float mu, float s1, float s2) {
    const float sigma = x < mu ? s1 : s2;
    const float t = (x - mu) / sigma;
    return alpha * expf(-0.5f * t * t);
}

bool finite_params(const kt_kerr_params& p) {
    return std::isfinite(p.rh) && std::isfinite(p.disk_inner);
}

}  // namespace

// =========================================================================================
extern "C" {

const char* kt_status_str(kt_status s) {
    switch (s) {
        case KT_OK: return "ok";
        case KT_ERR_INVALID_ARG: return "invalid argument";
        case KT_ERR_CUDA: return "CUDA error";
        case KT_ERR_LUT_OVERFLOW: return "colour temperature above lut_max_temp";
        case KT_ERR_NOT_READY: return "not ready";
        case KT_ERR_QUEUE_ORDER: return "frame queue out of order";
        case KT_ERR_NO_DEVICE: return "no CUDA device";
        case KT_ERR_UNSUPPORTED: return "unsupported";
        case KT_ERR_TIMEOUT: return "device wait timed out";
    }
    return "unknown status";
}
const char* kt_last_error(void) { return g_last_error.c_str(); }
int kt_abi_version(void) { return KT_ABI_VERSION; }

kt_status kt_config_default(kt_config* c) {
    if (!c) return fail(KT_ERR_INVALID_ARG, "cfg is NULL");
    std::memset(c, 0, sizeof *c);
    c->width = 2100;
    c->height = 900;
    c->block_dim[0] = 16;
    c->block_dim[1] = 16;
    c->bloom_enabled = 1;
    c->bloom_intensity = 0.5f;
    c->bloom_radius = 48.0f;
    c->lut_size = 4096;
    c->lut_max_temp = 3e4f;
    c->wavelength_start = 380.0f;
    c->wavelength_end = 720.0f;
    c->wavelength_step = 10.0f;
    c->use_fast_math = 1;
    c->spp = 4;
    c->exposure_scale = 3e-3f;
    c->sky_grid_divisions = 40;
    c->sky_line_thickness = 5e-4f;
    c->sky_intensity = 30.0f;
    c->spin = -0.45f;
    c->mass = 0.5f;
    c->disk_outer_radius = 40.0f;
    c->disk_temperature_scale = 3e4f;
    c->initial_step = 1.0f;
    c->tolerance = 1e-5f;
    c->max_steps = 100;
    c->max_attempts = 3;
    c->transmittance_cutoff = 1e-2f;
    c->horizon_epsilon = 5e-7f;
    c->escape_radius = 80.0f;
    c->noise_enabled = 1;
    c->noise_scale = 0.1f;
    c->noise_strength = 0.6f;
    c->noise_winding = 50.0f;
    c->noise_detail = 10;
    c->mode = KT_MODE_REF;
    c->precision = KT_PREC_FP32;
    c->photon_zone_factor = 1.5f;
    return KT_OK;
}

float kt_calc_isco(float a_norm, int prograde, float mass) { return isco_f32(a_norm, prograde != 0, mass); }

kt_status kt_build_kerr_params(const kt_config* cfg, kt_kerr_params* out) {
    if (!cfg || !out) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    if (cfg->width == 0) return fail(KT_ERR_INVALID_ARG, "window width must not be 0");
    if (cfg->height == 0) return fail(KT_ERR_INVALID_ARG, "window height must not be 0");
    const float spin = cfg->spin, mass = cfg->mass;
    if (!std::isfinite(spin)) return fail(KT_ERR_INVALID_ARG, "black hole spin is not finite: %g", spin);
    if (!std::isfinite(mass)) return fail(KT_ERR_INVALID_ARG, "black hole mass is not finite: %g", mass);
    if (mass == 0.0f) return fail(KT_ERR_INVALID_ARG, "black hole mass must not be 0");
    kt_kerr_params p;
    std::memset(&p, 0, sizeof p);
    p.a = spin;
    p.m = mass;
    p.inv_m = 1.0f / mass;
    p.aa = spin * spin;
    p.a_norm = spin * p.inv_m;
    p.rh = mass + sqrtf(fmaxf(fmaf(mass, mass, -p.aa), 0.0f));
    p.disk_inner = isco_f32(p.a_norm, true, mass);
    if (!finite_params(p)) return fail(KT_ERR_INVALID_ARG, "Kerr parameters are not finite");
    if (!std::isfinite(cfg->noise_scale)) return fail(KT_ERR_INVALID_ARG, "disk noise scale is not finite");
    if (!std::isfinite(cfg->noise_strength)) return fail(KT_ERR_INVALID_ARG, "disk noise strength is not finite");
    if (!std::isfinite(cfg->noise_winding)) return fail(KT_ERR_INVALID_ARG, "disk noise winding is not finite");
    if (cfg->noise_detail > (uint32_t)std::numeric_limits<int32_t>::max())
        return fail(KT_ERR_INVALID_ARG, "disk noise detail out of i32 range: %u", cfg->noise_detail);
    const double w = (double)cfg->width, h = (double)cfg->height;
    if (!f32_from_f64(w / h, &p.aspect_ratio) || !f32_from_f64(2.0 / w, &p.inv_w_2) ||
        !f32_from_f64(2.0 / h, &p.inv_h_2))
        return fail(KT_ERR_INVALID_ARG, "window size conversion failed");
    p.disk_noise_scale = cfg->noise_scale;
    p.disk_noise_strength = cfg->noise_strength;
    p.disk_noise_winding = cfg->noise_winding;
    p.disk_noise_enabled = cfg->noise_enabled ? 1 : 0;
    p.disk_noise_detail = (int32_t)cfg->noise_detail;
    *out = p;
    return KT_OK;
}

kt_status kt_generate_blackbody_lut(uint32_t size, float max_temp, float wl_start, float wl_end,
                                    float wl_step, float* out) {
    if (!out) return fail(KT_ERR_INVALID_ARG, "out is NULL");
    if (size < 2) return fail(KT_ERR_INVALID_ARG, "blackbody LUT size must be at least 2");
    if (!std::isfinite(wl_step) || wl_step <= 0.0f)
        return fail(KT_ERR_INVALID_ARG, "wavelength step must be positive and finite");
    std::vector<float> temps(size);
    for (uint32_t i = 0; i < size; ++i) {
        const double ratio = (double)i / (double)(size - 1);
        if (!f32_from_f64(ratio * (double)max_temp, &temps[i]))
            return fail(KT_ERR_INVALID_ARG, "temperature value conversion failed");
    }
    std::vector<float> lambdas;
    for (float l = wl_start;;) {
        if (l > wl_end) break;
        lambdas.push_back(l);
        l += wl_step;
        if (lambdas.size() > (1u << 24)) return fail(KT_ERR_INVALID_ARG, "wavelength grid too large");
    }
    const size_t n = lambdas.size();
    std::vector<float> xs(n), ys(n), zs(n), inv_l5(n);
    for (size_t i = 0; i < n; ++i) {
        const float l = lambdas[i];
        const float l2 = l * l;
        inv_l5[i] = 1.0f / (l * (l2 * l2));
        xs[i] = cmf_lobe(l, 1.056f, 599.8f, 37.9f, 31.0f) + cmf_lobe(l, 0.362f, 442.0f, 16.0f, 26.7f) +
                cmf_lobe(l, -0.065f, 501.1f, 20.4f, 26.2f);
        ys[i] = cmf_lobe(l, 0.821f, 568.8f, 46.9f, 40.5f) + cmf_lobe(l, 0.286f, 530.9f, 16.3f, 31.1f);
        zs[i] = cmf_lobe(l, 1.217f, 437.0f, 11.8f, 36.0f) + cmf_lobe(l, 0.681f, 459.0f, 26.2f, 13.8f);
    }
    const float c2 = 1.4388e7f;
    for (uint32_t ti = 0; ti < size; ++ti) {
        const float t = temps[ti];
        float* row = out + 4 * (size_t)ti;
        if (t == 0.0f) {
            row[0] = row[1] = row[2] = row[3] = 0.0f;
            continue;
        }
        float xsum = 0.0f, ysum = 0.0f, zsum = 0.0f;
        for (size_t i = 0; i < n; ++i) {
            float inten = 0.0f;
            if (t > 0.0f) {
                const float l = lambdas[i];
                const float expo = c2 / (l * t);
                if (!(expo > 80.0f)) inten = (inv_l5[i] / expm1f(expo)) * 1e15f;
            }
            xsum += inten * xs[i];
            ysum += inten * ys[i];
            zsum += inten * zs[i];
        }
        xsum *= wl_step;
        ysum *= wl_step;
        zsum *= wl_step;
        row[0] = fmaf(3.240454f, xsum, fmaf(-1.5371385f, ysum, -0.4985314f * zsum));
        row[1] = fmaf(-0.969266f, xsum, fmaf(1.8760108f, ysum, 0.041556f * zsum));
        row[2] = fmaf(0.0556434f, xsum, fmaf(-0.2040259f, ysum, 1.0572252f * zsum));
        row[3] = 0.0f;
    }
    return KT_OK;
}

kt_status kt_generate_blackbody_lut_device(uint32_t size, float max_temp, float wl_start, float wl_end,
                                           float wl_step, float* dev_out, void* stream) {
    if (!dev_out) return fail(KT_ERR_INVALID_ARG, "dev_out is NULL");
    if (size < 2) return fail(KT_ERR_INVALID_ARG, "blackbody LUT size must be at least 2");
    if (!std::isfinite(wl_step) || wl_step <= 0.0f)
        return fail(KT_ERR_INVALID_ARG, "wavelength step must be positive and finite");
    int n = 0;  // the host generator's grid: f32 accumulation from wl_start while <= wl_end
    for (float l = wl_start; !(l > wl_end); l += wl_step)
        if (++n > (1 << 24)) return fail(KT_ERR_INVALID_ARG, "wavelength grid too large");
    const cudaError_t e = ktd::launch_blackbody_lut(size, max_temp, wl_start, n, wl_step,
                                                    reinterpret_cast<float4*>(dev_out), (cudaStream_t)stream);
    if (e != cudaSuccess) return cuda_fail(e, "blackbody LUT launch");
    return KT_OK;
}

kt_status kt_generate_disk_lut_device(const kt_kerr_params* p, float disk_outer, uint32_t size, float* dev_out,
                                      void* stream) {
    if (!p || !dev_out) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    if (size < 2) return fail(KT_ERR_INVALID_ARG, "disk temperature LUT size must be at least 2");
    if (!std::isfinite(disk_outer) || !std::isfinite(p->disk_inner) || disk_outer <= p->disk_inner)
        return fail(KT_ERR_INVALID_ARG, "disk radii must be finite with outer > inner: outer=%g, inner=%g",
                    disk_outer, p->disk_inner);
    const cudaError_t e = ktd::launch_disk_lut(size, p->a_norm, p->inv_m, p->disk_inner, disk_outer, dev_out,
                                               (cudaStream_t)stream);
    if (e != cudaSuccess) return cuda_fail(e, "disk LUT launch");
    return KT_OK;
}

kt_status kt_generate_disk_lut(const kt_kerr_params* p, float disk_outer, uint32_t size, float* out) {
    if (!p || !out) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    if (size < 2) return fail(KT_ERR_INVALID_ARG, "disk temperature LUT size must be at least 2");
    if (!std::isfinite(disk_outer)) return fail(KT_ERR_INVALID_ARG, "disk outer radius is not finite");
    if (!std::isfinite(p->disk_inner)) return fail(KT_ERR_INVALID_ARG, "disk inner radius is not finite");
    if (disk_outer <= p->disk_inner)
        return fail(KT_ERR_INVALID_ARG, "disk outer radius must exceed the inner radius: outer=%g, inner=%g",
                    disk_outer, p->disk_inner);
    const double inner = (double)p->disk_inner;
    const double span = (double)(disk_outer - p->disk_inner);
    const NtTerms terms = nt_terms_f32(p->a_norm, p->disk_inner, p->inv_m);
    for (uint32_t i = 0; i < size; ++i) {
        const double ratio = (double)i / (double)(size - 1);
        float r;
        if (!f32_from_f64(std::fma(ratio, span, inner), &r)) return fail(KT_ERR_INVALID_ARG, "disk radius conversion failed");
        const float f = nt_factor_f32(r, p->a_norm, p->disk_inner, p->inv_m, terms);
        if (!std::isfinite(f)) return fail(KT_ERR_INVALID_ARG, "disk flux factor is not finite");
        const float v = sqrtf(sqrtf(f));
        if (!std::isfinite(v)) return fail(KT_ERR_INVALID_ARG, "disk temperature factor is not finite");
        out[i] = v;
    }
    return KT_OK;
}

kt_status kt_build_defines(const kt_config* cfg, char* buf, size_t cap, size_t* len) {
    if (!cfg) return fail(KT_ERR_INVALID_ARG, "cfg is NULL");
    std::string s;
    char line[160];
    const struct { const char* k; uint32_t v; } ints[] = {
        {"CONFIG_SPP", cfg->spp},
        {"CONFIG_SKY_GRID_DIVISIONS", cfg->sky_grid_divisions},
        {"CONFIG_INTEGRATOR_MAX_STEPS", cfg->max_steps},
        {"CONFIG_INTEGRATOR_MAX_ATTEMPTS", cfg->max_attempts},
    };
    for (auto& e : ints) {
        snprintf(line, sizeof line, "#define %s %u\n", e.k, e.v);
        s += line;
    }
    const struct { const char* k; float v; } floats[] = {
        {"CONFIG_EXPOSURE_SCALE", cfg->exposure_scale},
        {"CONFIG_SKY_LINE_THICKNESS", cfg->sky_line_thickness},
        {"CONFIG_SKY_INTENSITY", cfg->sky_intensity},
        {"CONFIG_DISK_OUTER_RADIUS", cfg->disk_outer_radius},
        {"CONFIG_DISK_TEMPERATURE_SCALE", cfg->disk_temperature_scale},
        {"CONFIG_INTEGRATOR_INITIAL_STEP", cfg->initial_step},
        {"CONFIG_INTEGRATOR_TOLERANCE", cfg->tolerance},
        {"CONFIG_TRANSMITTANCE_CUTOFF", cfg->transmittance_cutoff},
        {"CONFIG_HORIZON_EPSILON", cfg->horizon_epsilon},
        {"CONFIG_ESCAPE_RADIUS", cfg->escape_radius},
        {"CONFIG_BLACKBODY_WAVELENGTH_STEP", cfg->wavelength_step},
    };
    for (auto& e : floats) {
        snprintf(line, sizeof line, "#define %s %.10f\n", e.k, (double)e.v);
        s += line;
    }
    if (len) *len = s.size();
    if (buf) {
        if (cap < s.size() + 1) return fail(KT_ERR_INVALID_ARG, "buffer too small (%zu < %zu)", cap, s.size() + 1);
        std::memcpy(buf, s.c_str(), s.size() + 1);
    }
    return KT_OK;
}

static void vnormalize(float v[3]) {
    const float len = sqrtf((v[0] * v[0] + v[1] * v[1]) + v[2] * v[2]);
    const float inv = 1.0f / len;
    v[0] *= inv;
    v[1] *= inv;
    v[2] *= inv;
}
static void vcross(const float a[3], const float b[3], float o[3]) {
    o[0] = a[1] * b[2] - b[1] * a[2];
    o[1] = a[2] * b[0] - b[2] * a[0];
    o[2] = a[0] * b[1] - b[0] * a[1];
}
static const float kRadsPerDeg = 3.14159265358979323846f / 180.0f;  // f32::to_radians

kt_status kt_camera_basis(float yaw_deg, float pitch_deg, float fwd[3], float rgt[3], float up[3]) {
    if (!fwd || !rgt || !up) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    const float yaw = yaw_deg * kRadsPerDeg, pitch = pitch_deg * kRadsPerDeg;
    float f[3] = {sinf(yaw) * cosf(pitch), sinf(pitch), -cosf(yaw) * cosf(pitch)};
    vnormalize(f);
    const float world_up[3] = {0.0f, 1.0f, 0.0f};
    float r[3], u[3];
    vcross(f, world_up, r);
    vnormalize(r);
    vcross(r, f, u);
    vnormalize(u);
    for (int i = 0; i < 3; ++i) {
        fwd[i] = f[i];
        rgt[i] = r[i];
        up[i] = u[i];
    }
    return KT_OK;
}

float kt_fov_scale(float fov_deg) { return tanf((fov_deg * kRadsPerDeg) / 2.0f); }

kt_status kt_validate_bloom(const kt_config* cfg, int32_t* enabled, float* intensity, float* radius,
                            int32_t* radius_int) {
    if (!cfg) return fail(KT_ERR_INVALID_ARG, "cfg is NULL");
    const float inten = cfg->bloom_intensity;
    if (!std::isfinite(inten) || inten < 0.0f) return fail(KT_ERR_INVALID_ARG, "invalid bloom intensity: %g", inten);
    const float rad = cfg->bloom_radius;
    if (!std::isfinite(rad) || rad < 0.0f) return fail(KT_ERR_INVALID_ARG, "invalid bloom radius: %g", rad);
    const double max_r = (double)std::numeric_limits<int32_t>::max();
    if ((double)rad > max_r) return fail(KT_ERR_INVALID_ARG, "bloom radius too large: %g", rad);
    int32_t ri = 0;
    if (rad > 0.0f) {
        const float c = ceilf(rad);
        if ((double)c > max_r) return fail(KT_ERR_INVALID_ARG, "bloom radius too large: %g", rad);
        ri = (int32_t)c;
    }
    if (enabled) *enabled = cfg->bloom_enabled ? 1 : 0;
    if (intensity) *intensity = inten;
    if (radius) *radius = rad;
    if (radius_int) *radius_int = ri;
    return KT_OK;
}

}  // extern "C"

// =========================================================================================
// Device context
// =========================================================================================
// struct kt_context is defined in kt_context.h (shared with the autotuner, kt_tune.cpp).

namespace {

void destroy_ctx(kt_context* c) {
    if (!c) return;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(c->device);
    if (c->bb_tex) cudaDestroyTextureObject(c->bb_tex);
    if (c->disk_tex) cudaDestroyTextureObject(c->disk_tex);
    if (c->bb_array) cudaFreeArray(c->bb_array);
    if (c->disk_array) cudaFreeArray(c->disk_array);
    cudaFree(c->bb_lut_dev);
    cudaFree(c->disk_lut_dev);
    cudaFree(c->queue);
    cudaFree(c->counters);
    cudaFree(c->order);
    cudaFree(c->bloom_scratch);
    cudaFree(c->post_tables);
    cudaSetDevice(prev);
    delete c;
}

// 1D cudaArray + texture object with the reference's sampler (texture.rs:86-202): float
// channels, linear filtering, normalised coordinates, clamp addressing.  The blackbody LUT is
// allocated with height 1, the disk LUT with height 0, as in texture.rs:37-67.
kt_status make_lut_texture(const float* host, uint32_t n, int channels, size_t height,
                           cudaArray_t* arr, cudaTextureObject_t* tex,
                           cudaMemcpyKind kind = cudaMemcpyHostToDevice) {
    const cudaChannelFormatDesc desc =
        channels == 4 ? cudaCreateChannelDesc(32, 32, 32, 32, cudaChannelFormatKindFloat)
                      : cudaCreateChannelDesc(32, 0, 0, 0, cudaChannelFormatKindFloat);
    KT_CUDA(cudaMallocArray(arr, &desc, n, height, cudaArrayDefault), "cudaMallocArray");
    const size_t row_bytes = (size_t)n * channels * sizeof(float);
    KT_CUDA(cudaMemcpy2DToArray(*arr, 0, 0, host, row_bytes, row_bytes, 1, kind), "copy LUT to CUDA array");
    cudaResourceDesc rd;
    std::memset(&rd, 0, sizeof rd);
    rd.resType = cudaResourceTypeArray;
    rd.res.array.array = *arr;
    cudaTextureDesc td;
    std::memset(&td, 0, sizeof td);
    td.addressMode[0] = td.addressMode[1] = td.addressMode[2] = cudaAddressModeClamp;
    td.filterMode = cudaFilterModeLinear;
    td.readMode = cudaReadModeElementType;
    td.normalizedCoords = 1;
    KT_CUDA(cudaCreateTextureObject(tex, &rd, &td, nullptr), "cudaCreateTextureObject");
    return KT_OK;
}

kt_status fill_scene(kt_context* c) {
    const kt_config& cfg = c->cfg;
    const kt_kerr_params& p = c->params;
    ktd::Scene& s = c->scene;
    std::memset(&s, 0, sizeof s);
    s.a = p.a; s.M = p.m; s.aa = p.aa; s.inv_M = p.inv_m; s.a_norm = p.a_norm; s.rh = p.rh;
    s.disk_inner = p.disk_inner;
    s.disk_outer = cfg.disk_outer_radius;
    s.disk_inner_d = (double)s.disk_inner;
    s.disk_outer_d = (double)s.disk_outer;
    s.disk_lut_d = nullptr;
    s.inv_w_2 = p.inv_w_2; s.inv_h_2 = p.inv_h_2; s.aspect = p.aspect_ratio;
    s.noise_scale = p.disk_noise_scale; s.noise_strength = p.disk_noise_strength;
    s.noise_winding = p.disk_noise_winding; s.noise_enabled = p.disk_noise_enabled;
    s.noise_detail = p.disk_noise_detail;
    const uint32_t imax = (uint32_t)std::numeric_limits<int32_t>::max();
    if (cfg.spp > imax || cfg.max_steps > imax || cfg.max_attempts > imax || cfg.sky_grid_divisions > imax)
        return fail(KT_ERR_INVALID_ARG, "integer knob out of i32 range");
    if (cfg.max_attempts == 0) return fail(KT_ERR_INVALID_ARG, "max_attempts must be at least 1");
    s.spp = (int)cfg.spp;
    s.max_steps = (int)cfg.max_steps;
    s.max_attempts = (int)cfg.max_attempts;
    s.sky_div = (int)cfg.sky_grid_divisions;
    s.sky_spacing = 3.14159265f / (float)cfg.sky_grid_divisions;
    const double d_exposure = define_value(cfg.exposure_scale);
    const double d_thick = define_value(cfg.sky_line_thickness);
    const double d_sky = define_value(cfg.sky_intensity);
    const double d_temp = define_value(cfg.disk_temperature_scale);
    const double d_h0 = define_value(cfg.initial_step);
    const double d_tol = define_value(cfg.tolerance);
    const double d_cut = define_value(cfg.transmittance_cutoff);
    const double d_heps = define_value(cfg.horizon_epsilon);
    const double d_esc = define_value(cfg.escape_radius);
    const double d_wl = define_value(cfg.wavelength_step);
    s.h0 = (float)d_h0;
    s.base_tol = (float)d_tol;
    s.sky_thickness = (float)d_thick;
    s.horizon_lt = float_ceil((double)p.rh + d_heps);
    s.escape_gt = float_floor(d_esc);
    s.cutoff_gt = float_floor(d_cut);
    const float inv_spp = 1.0f / (float)cfg.spp;
    s.final_scale = (float)(d_exposure * (double)inv_spp);
    s.sample_first = 0;
    s.pixel_centre = (cfg.mode == KT_MODE_SPEC && cfg.spp == 1) ? 1 : 0;
    s.accum = nullptr;
    s.temp_scale = d_temp;
    s.wl_step = d_wl;
    s.sky_intensity = d_sky;
    s.a_d = (double)p.a;
    s.aa_d = s.a_d * s.a_d;
    s.M_d = (double)p.m;
    const double rh_d = s.M_d + std::sqrt(std::fmax(s.M_d * s.M_d - s.aa_d, 0.0));
    s.horizon_d = (double)p.rh + d_heps;  // the reference adds the define to the f32 rh
    (void)rh_d;
    s.escape_d = d_esc;
    s.cutoff_d = d_cut;
    s.h0_d = d_h0;
    s.base_tol_d = d_tol;
    s.bb_tex = c->bb_tex;
    s.disk_tex = c->disk_tex;
    s.bb_lut = c->bb_lut_dev;
    s.disk_lut = c->disk_lut_dev;
    s.lut_size = (int)cfg.lut_size;
    s.lut_max_temp = cfg.lut_max_temp;
    s.mode = cfg.mode;
    s.precision = cfg.precision;
    s.noise_seed = cfg.noise_seed;
    s.noise_phase = cfg.noise_phase;
    const float zf = cfg.photon_zone_factor > 0.0f ? cfg.photon_zone_factor : 1.5f;
    // retrograde equatorial photon orbit r_ph = 2M (1 + cos(2/3 acos(|a|/M))): 3M for a = 0,
    // 4M for |a| = M; the prograde orbit lies inside it
    const double an = std::fmin(std::fabs((double)p.a_norm), 1.0);
    const double rph = 2.0 * s.M_d * (1.0 + std::cos(2.0 / 3.0 * std::acos(an)));
    s.zone_r = (float)(zf * rph);
    s.zone_err64 = cfg.tolerance < 3e-7f ? 1 : 0;
    s.spec_tol_floor = 1.0f;
    s.width = (int)cfg.width;
    s.height = (int)cfg.height;
    return KT_OK;
}

kt_status fill_post(kt_context* c) {
    int32_t en = 0, ri = 0;
    float inten = 0.0f, rad = 0.0f;
    kt_status st = kt_validate_bloom(&c->cfg, &en, &inten, &rad, &ri);
    if (st != KT_OK) return st;
    ktd::PostParams& pp = c->post;
    pp.width = (int)c->cfg.width;
    pp.height = (int)c->cfg.height;
    pp.radius = ri;
    pp.sigma = rad / 3.0f;
    pp.intensity = inten;
    pp.active = (en && ri > 0 && inten > 0.0f) ? 1 : 0;
    pp.mode = c->cfg.mode;
    pp.threshold = c->cfg.bloom_threshold;
    return KT_OK;
}

kt_status validate_cfg(const kt_config* cfg) {
    if (!cfg) return fail(KT_ERR_INVALID_ARG, "cfg is NULL");
    if (!cfg->use_fast_math) return fail(KT_ERR_UNSUPPORTED, "the kernels are built with use_fast_math; use_fast_math=false is not available");
    if (cfg->mode != KT_MODE_REF && cfg->mode != KT_MODE_SPEC) return fail(KT_ERR_INVALID_ARG, "unknown mode %d", cfg->mode);
    if (cfg->precision < KT_PREC_FP32 || cfg->precision > KT_PREC_FP64) return fail(KT_ERR_INVALID_ARG, "unknown precision %d", cfg->precision);
    if (cfg->mode == KT_MODE_REF && cfg->precision != KT_PREC_FP32)
        return fail(KT_ERR_INVALID_ARG, "reference mode runs the reference's FP32 arithmetic; use KT_MODE_SPEC for mixed/FP64");
    if (cfg->width == 0 || cfg->height == 0)
        return fail(KT_ERR_INVALID_ARG, "empty image: %ux%u", cfg->width, cfg->height);
    if (cfg->width > 32768 || cfg->height > 32768)
        return fail(KT_ERR_INVALID_ARG, "image too large: %ux%u", cfg->width, cfg->height);
    const uint64_t bt = (uint64_t)cfg->block_dim[0] * cfg->block_dim[1];
    if (cfg->block_dim[0] == 0 || cfg->block_dim[1] == 0 || bt > 1024)
        return fail(KT_ERR_INVALID_ARG, "block_dim %ux%u must be non-zero with at most 1024 threads",
                    cfg->block_dim[0], cfg->block_dim[1]);
    if (cfg->lut_size < 2) return fail(KT_ERR_INVALID_ARG, "lut_size must be at least 2");
    if (!std::isfinite(cfg->lut_max_temp)) return fail(KT_ERR_INVALID_ARG, "lut_max_temp is not finite");
    return KT_OK;
}

// device_luts: both tables are generated on the device (kt_generate_*_lut_device, on the legacy
// default stream) and the textures are filled from there.
kt_status create_impl(const kt_config* cfg, int device, const float* bb_in, const float* disk_in,
                      uint32_t lut_n, kt_context** out, bool device_luts = false) {
    if (!out) return fail(KT_ERR_INVALID_ARG, "out is NULL");
    *out = nullptr;
    kt_status st = validate_cfg(cfg);
    if (st != KT_OK) return st;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) return fail(KT_ERR_NO_DEVICE, "no CUDA device");
    if (device < 0 || device >= ndev) return fail(KT_ERR_INVALID_ARG, "device %d out of range", device);
    kt_context* c = new (std::nothrow) kt_context();
    if (!c) return fail(KT_ERR_INVALID_ARG, "out of host memory");
    c->device = device;
    c->cfg = *cfg;
    c->block_x = (int)cfg->block_dim[0];
    c->block_y = (int)cfg->block_dim[1];
    auto bail = [&](kt_status s) { destroy_ctx(c); return s; };
    if ((st = kt_build_kerr_params(cfg, &c->params)) != KT_OK) return bail(st);
    if ((st = fill_post(c)) != KT_OK) return bail(st);
    const uint32_t n = cfg->lut_size;
    std::vector<float> bb, disk;
    if (bb_in) {
        if (lut_n != n) return bail(fail(KT_ERR_INVALID_ARG, "LUT length %u does not match lut_size %u", lut_n, n));
        bb.assign(bb_in, bb_in + 4 * (size_t)n);
        disk.assign(disk_in, disk_in + n);
    } else if (!device_luts) {
        bb.resize(4 * (size_t)n);
        disk.resize(n);
        if ((st = kt_generate_blackbody_lut(n, cfg->lut_max_temp, cfg->wavelength_start, cfg->wavelength_end,
                                            cfg->wavelength_step, bb.data())) != KT_OK)
            return bail(st);
        if ((st = kt_generate_disk_lut(&c->params, cfg->disk_outer_radius, n, disk.data())) != KT_OK) return bail(st);
    }
    int prev = 0;
    cudaGetDevice(&prev);
    if (cudaSetDevice(device) != cudaSuccess) return bail(fail(KT_ERR_CUDA, "cudaSetDevice(%d) failed", device));
    auto step = [&](kt_status s) { if (s != KT_OK) { cudaSetDevice(prev); destroy_ctx(c); } return s; };
    cudaError_t e;
    if ((e = cudaMalloc(&c->bb_lut_dev, 4 * (size_t)n * sizeof(float))) != cudaSuccess ||
        (e = cudaMalloc(&c->disk_lut_dev, (size_t)n * sizeof(float))) != cudaSuccess)
        return step(cuda_fail(e, "context LUT allocation"));
    if (device_luts) {
        if ((st = step(kt_generate_blackbody_lut_device(n, cfg->lut_max_temp, cfg->wavelength_start, cfg->wavelength_end,
                                                        cfg->wavelength_step, reinterpret_cast<float*>(c->bb_lut_dev),
                                                        nullptr))) != KT_OK ||
            (st = step(kt_generate_disk_lut_device(&c->params, cfg->disk_outer_radius, n, c->disk_lut_dev, nullptr))) !=
                KT_OK)
            return st;
        if ((e = cudaDeviceSynchronize()) != cudaSuccess) return step(cuda_fail(e, "device LUT generation"));
        const float* bbd = reinterpret_cast<const float*>(c->bb_lut_dev);
        if ((st = step(make_lut_texture(bbd, n, 4, 1, &c->bb_array, &c->bb_tex, cudaMemcpyDeviceToDevice))) != KT_OK)
            return st;
        if ((st = step(make_lut_texture(c->disk_lut_dev, n, 1, 0, &c->disk_array, &c->disk_tex, cudaMemcpyDeviceToDevice))) !=
            KT_OK)
            return st;
    } else {
        if ((st = step(make_lut_texture(bb.data(), n, 4, 1, &c->bb_array, &c->bb_tex))) != KT_OK) return st;
        if ((st = step(make_lut_texture(disk.data(), n, 1, 0, &c->disk_array, &c->disk_tex))) != KT_OK) return st;
        if ((e = cudaMemcpy(c->bb_lut_dev, bb.data(), bb.size() * sizeof(float), cudaMemcpyHostToDevice)) != cudaSuccess ||
            (e = cudaMemcpy(c->disk_lut_dev, disk.data(), disk.size() * sizeof(float), cudaMemcpyHostToDevice)) !=
                cudaSuccess)
            return step(cuda_fail(e, "LUT upload"));
    }
    if ((e = cudaMalloc(&c->queue, 64)) != cudaSuccess ||
        (e = cudaMalloc(&c->counters, 8 * sizeof(unsigned long long))) != cudaSuccess ||
        (c->post.active &&
         (e = cudaMalloc(&c->bloom_scratch, ktd::post_scratch_bytes((int)cfg->width, (int)cfg->height))) != cudaSuccess) ||
        (e = cudaMalloc(&c->post_tables, ktd::post_table_floats(c->post) * sizeof(float) + 16)) != cudaSuccess)
        return step(cuda_fail(e, "context allocation"));
    // the tables are complete before the context is handed out: its calls may come on any stream
    if ((e = ktd::launch_post_tables(c->post, c->post_tables, nullptr)) != cudaSuccess ||
        (e = cudaStreamSynchronize(nullptr)) != cudaSuccess)
        return step(cuda_fail(e, "blur tables"));
    if ((st = step(fill_scene(c))) != KT_OK) return st;
    cudaSetDevice(prev);
    *out = c;
    return KT_OK;
}

}  // namespace

namespace ktd {
// Device-side scene constants of a config without a context (the LUT pointers and texture
// objects are left empty for the caller to fill).
kt_status scene_from_config(const kt_config* cfg, Scene* out) {
    kt_status st = validate_cfg(cfg);
    if (st != KT_OK) return st;
    kt_context tmp;
    tmp.cfg = *cfg;
    if ((st = kt_build_kerr_params(cfg, &tmp.params)) != KT_OK) return st;
    if ((st = fill_scene(&tmp)) != KT_OK) return st;
    *out = tmp.scene;
    return KT_OK;
}
kt_status set_error(kt_status s, const char* msg) { return fail(s, "%s", msg); }
}  // namespace ktd

namespace {

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        cudaGetDevice(&prev);
        if (prev != dev) cudaSetDevice(dev); else prev = -1;
    }
    ~DeviceGuard() { if (prev >= 0) cudaSetDevice(prev); }
};

int plain_bx(const kt_context* c) { return c->tuning.block_x > 0 ? c->tuning.block_x : c->block_x; }
int plain_by(const kt_context* c) { return c->tuning.block_y > 0 ? c->tuning.block_y : c->block_y; }
unsigned* order_buffer(const kt_context* c) { return c->tuning.order == KT_ORDER_LONG_FIRST ? c->order : nullptr; }

ktd::Camera to_camera(const kt_camera* cam) {
    ktd::Camera c;
    for (int i = 0; i < 3; ++i) {
        c.pos[i] = cam->cam_pos[i];
        c.fwd[i] = cam->fwd[i];
        c.rgt[i] = cam->rgt[i];
        c.up[i] = cam->up[i];
    }
    c.fov_scale = cam->fov_scale;
    return c;
}

}  // namespace

extern "C" {

kt_status kt_context_create(const kt_config* cfg, int device, kt_context** out) {
    return create_impl(cfg, device, nullptr, nullptr, 0, out);
}
kt_status kt_context_create_device_luts(const kt_config* cfg, int device, kt_context** out) {
    return create_impl(cfg, device, nullptr, nullptr, 0, out, true);
}
kt_status kt_context_create_with_luts(const kt_config* cfg, int device, const float* bb_rgba,
                                      const float* disk, uint32_t lut_n, kt_context** out) {
    if (!bb_rgba || !disk) return fail(KT_ERR_INVALID_ARG, "LUT pointer is NULL");
    return create_impl(cfg, device, bb_rgba, disk, lut_n, out);
}
void kt_context_destroy(kt_context* ctx) { destroy_ctx(ctx); }
kt_status kt_context_params(const kt_context* ctx, kt_kerr_params* out) {
    if (!ctx || !out) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    *out = ctx->params;
    return KT_OK;
}

kt_status kt_context_set_tuning(kt_context* ctx, const kt_tuning* t) {
    if (!ctx || !t) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    if (t->schedule != KT_SCHED_PLAIN && t->schedule != KT_SCHED_WAVEFRONT)
        return fail(KT_ERR_INVALID_ARG, "tuning schedule %d must be plain or wavefront", t->schedule);
    if (t->blocks_per_sm < 3 || t->blocks_per_sm > 6) return fail(KT_ERR_INVALID_ARG, "blocks_per_sm %d not in 3..6", t->blocks_per_sm);
    if (t->refill_min < 1 || t->refill_min > 32) return fail(KT_ERR_INVALID_ARG, "refill_min %d not in 1..32", t->refill_min);
    if (t->block_x < 0 || t->block_y < 0 || (int64_t)t->block_x * t->block_y > 1024 ||
        ((t->block_x == 0) != (t->block_y == 0)))
        return fail(KT_ERR_INVALID_ARG, "plain block %dx%d invalid", t->block_x, t->block_y);
    if (t->order != KT_ORDER_TILES && t->order != KT_ORDER_LONG_FIRST)
        return fail(KT_ERR_INVALID_ARG, "tuning order %d must be tiles or long-first", t->order);
    if (t->keep_frozen != 0 && t->keep_frozen != 1)
        return fail(KT_ERR_INVALID_ARG, "tuning keep_frozen %d must be 0 or 1", t->keep_frozen);
    if (t->order == KT_ORDER_LONG_FIRST && !ctx->order) {
        DeviceGuard g(ctx->device);
        const size_t words = ktd::kOrderHeader + (size_t)ctx->cfg.width * ctx->cfg.height;
        KT_CUDA(cudaMalloc(&ctx->order, words * sizeof(unsigned)), "allocate pixel order");
    }
    ctx->tuning.order = t->order;
    ctx->tuning.schedule = t->schedule;
    ctx->tuning.block_x = t->block_x;
    ctx->tuning.block_y = t->block_y;
    ctx->tuning.blocks_per_sm = t->blocks_per_sm;
    ctx->tuning.refill_min = t->refill_min;
    ctx->tuning.keep_frozen = t->keep_frozen;
    ctx->scene.keep_frozen = t->keep_frozen;
    return KT_OK;
}
kt_status kt_context_get_tuning(const kt_context* ctx, kt_tuning* t) {
    if (!ctx || !t) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    t->schedule = ctx->tuning.schedule;
    t->block_x = ctx->tuning.block_x;
    t->block_y = ctx->tuning.block_y;
    t->blocks_per_sm = ctx->tuning.blocks_per_sm;
    t->refill_min = ctx->tuning.refill_min;
    t->order = ctx->tuning.order;
    t->keep_frozen = ctx->tuning.keep_frozen;
    return KT_OK;
}

kt_status kt_trace(kt_context* ctx, void* stream, const kt_camera* cam, int32_t schedule,
                   float* hdr_out, uint32_t* err_word) {
    if (!ctx || !cam || !hdr_out || !err_word) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    if (schedule < KT_SCHED_PLAIN || schedule > KT_SCHED_AUTO) return fail(KT_ERR_INVALID_ARG, "unknown schedule %d", schedule);
    DeviceGuard g(ctx->device);
    const int sched = schedule == KT_SCHED_AUTO ? ctx->tuning.schedule : schedule;
    const cudaError_t e = ktd::launch_trace(ctx->scene, to_camera(cam), sched, reinterpret_cast<float4*>(hdr_out),
                                            err_word, ctx->queue, nullptr, nullptr, ctx->tuning, plain_bx(ctx),
                                            plain_by(ctx), order_buffer(ctx), (cudaStream_t)stream);
    if (e != cudaSuccess) return cuda_fail(e, "trace launch");
    return KT_OK;
}

kt_status kt_trace_counted(kt_context* ctx, void* stream, const kt_camera* cam, int32_t schedule,
                           float* hdr_out, uint32_t* err_word, kt_trace_stats* stats, float* aux_out) {
    if (!ctx || !cam || !hdr_out || !err_word || !stats) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    if (schedule < KT_SCHED_PLAIN || schedule > KT_SCHED_AUTO) return fail(KT_ERR_INVALID_ARG, "unknown schedule %d", schedule);
    DeviceGuard g(ctx->device);
    const int sched = schedule == KT_SCHED_AUTO ? ctx->tuning.schedule : schedule;
    cudaStream_t st = (cudaStream_t)stream;
    KT_CUDA(cudaMemsetAsync(ctx->counters, 0, 8 * sizeof(unsigned long long), st), "clear counters");
    if (aux_out)  // all-ones words are NaN: pixels without a traced sample 0 stay NaN
        KT_CUDA(cudaMemsetAsync(aux_out, 0xff, (size_t)ctx->cfg.width * ctx->cfg.height * 4 * sizeof(float), st),
                "clear aux");
    cudaError_t e = ktd::launch_trace(ctx->scene, to_camera(cam), sched, reinterpret_cast<float4*>(hdr_out),
                                      err_word, ctx->queue, ctx->counters, reinterpret_cast<float4*>(aux_out),
                                      ctx->tuning, plain_bx(ctx), plain_by(ctx), order_buffer(ctx), st);
    if (e != cudaSuccess) return cuda_fail(e, "trace launch");
    unsigned long long h[8];
    KT_CUDA(cudaMemcpyAsync(h, ctx->counters, sizeof h, cudaMemcpyDeviceToHost, st), "read counters");
    KT_CUDA(cudaStreamSynchronize(st), "synchronise");
    stats->rays = h[0];
    stats->steps = h[1];
    stats->attempts = h[2];
    stats->rhs_evals = h[3];
    stats->frozen_rays = h[4];
    stats->fp64_steps = h[5];
    return KT_OK;
}

kt_status kt_trace_progressive(kt_context* ctx, void* stream, const kt_camera* cam, uint32_t first_sample,
                               uint32_t n_samples, float* accum, float* hdr_out, uint32_t* err_word) {
    if (!ctx || !cam || !accum || !hdr_out || !err_word) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    if (n_samples == 0) return fail(KT_ERR_INVALID_ARG, "n_samples must be at least 1");
    if ((uint64_t)first_sample + n_samples > (uint64_t)std::numeric_limits<int32_t>::max())
        return fail(KT_ERR_INVALID_ARG, "sample range out of i32 range");
    DeviceGuard g(ctx->device);
    ktd::Scene sc = ctx->scene;
    sc.sample_first = (int)first_sample;
    sc.spp = (int)n_samples;
    sc.pixel_centre = 0;
    sc.accum = reinterpret_cast<float4*>(accum);
    // kernel.cu:105,136 for the total sample count so far
    const float inv_spp = 1.0f / (float)(first_sample + n_samples);
    sc.final_scale = (float)(define_value(ctx->cfg.exposure_scale) * (double)inv_spp);
    const cudaError_t e = ktd::launch_trace(sc, to_camera(cam), KT_SCHED_PLAIN, reinterpret_cast<float4*>(hdr_out),
                                            err_word, ctx->queue, nullptr, nullptr, ctx->tuning, plain_bx(ctx),
                                            plain_by(ctx), nullptr, (cudaStream_t)stream);
    if (e != cudaSuccess) return cuda_fail(e, "trace launch");
    return KT_OK;
}

kt_status kt_fma_peak(int device, uint32_t iters, double* tflops, float* ms) {
    if (!tflops) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    if (iters == 0 || iters > (1u << 24)) return fail(KT_ERR_INVALID_ARG, "iters out of range");
    DeviceGuard g(device);
    int sms = 0, per_sm = 0;
    KT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "SM count");
    KT_CUDA(cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxThreadsPerMultiProcessor, device), "threads per SM");
    const int blocks = sms * std::max(1, per_sm / 512);
    float* sink = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaStream_t st = nullptr;
    kt_status out = KT_OK;
    float best = 0.0f;
    do {
        cudaError_t e;
        if ((e = cudaMalloc(&sink, sizeof(float))) != cudaSuccess || (e = cudaEventCreate(&e0)) != cudaSuccess ||
            (e = cudaEventCreate(&e1)) != cudaSuccess ||
            (e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking)) != cudaSuccess ||
            (e = ktd::launch_fma_probe(blocks, (int)iters, sink, st)) != cudaSuccess ||
            (e = cudaStreamSynchronize(st)) != cudaSuccess) {
            out = cuda_fail(e, "FMA probe");
            break;
        }
        for (int rep = 0; rep < 5 && out == KT_OK; ++rep) {
            float t = 0.0f;
            if ((e = cudaEventRecord(e0, st)) != cudaSuccess ||
                (e = ktd::launch_fma_probe(blocks, (int)iters, sink, st)) != cudaSuccess ||
                (e = cudaEventRecord(e1, st)) != cudaSuccess || (e = cudaEventSynchronize(e1)) != cudaSuccess ||
                (e = cudaEventElapsedTime(&t, e0, e1)) != cudaSuccess) {
                out = cuda_fail(e, "FMA probe timing");
                break;
            }
            if (best == 0.0f || t < best) best = t;
        }
    } while (false);
    if (sink) cudaFree(sink);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (st) cudaStreamDestroy(st);
    if (out != KT_OK) return out;
    const double flops = 16.0 * (double)iters * (double)blocks * 512.0;
    *tflops = flops / ((double)best * 1e-3) / 1e12;
    if (ms) *ms = best;
    return KT_OK;
}

static bool misaligned(const void* p, uintptr_t a) { return ((uintptr_t)p & (a - 1)) != 0; }

kt_status kt_bloom_horizontal(kt_context* ctx, void* stream, const float* hdr, float* bloom) {
    if (!ctx || !hdr || !bloom) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    if (misaligned(hdr, 16) || misaligned(bloom, 16)) return fail(KT_ERR_INVALID_ARG, "hdr and bloom must be 16-byte aligned");
    DeviceGuard g(ctx->device);
    const cudaError_t e = ktd::launch_bloom_horizontal(ctx->post, reinterpret_cast<const float4*>(hdr),
                                                       reinterpret_cast<float4*>(bloom), (cudaStream_t)stream);
    if (e != cudaSuccess) return cuda_fail(e, "bloom launch");
    return KT_OK;
}

kt_status kt_post_process(kt_context* ctx, void* stream, const float* hdr, const float* bloom, uint32_t* image_out) {
    if (!ctx || !hdr || !image_out || (ctx->post.active && !bloom)) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    if (misaligned(hdr, 16) || misaligned(bloom, 16) || misaligned(image_out, 4))
        return fail(KT_ERR_INVALID_ARG, "hdr and bloom must be 16-byte aligned, image_out 4-byte aligned");
    DeviceGuard g(ctx->device);
    const cudaError_t e = ktd::launch_post_process(ctx->post, reinterpret_cast<const float4*>(hdr),
                                                   reinterpret_cast<const float4*>(bloom), image_out,
                                                   (cudaStream_t)stream);
    if (e != cudaSuccess) return cuda_fail(e, "post launch");
    return KT_OK;
}

kt_status kt_post_fused(kt_context* ctx, void* stream, const float* hdr, uint32_t* image_out) {
    if (!ctx || !hdr || !image_out) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    if (misaligned(hdr, 16) || misaligned(image_out, 4))
        return fail(KT_ERR_INVALID_ARG, "hdr must be 16-byte aligned, image_out 4-byte aligned");
    DeviceGuard g(ctx->device);
    const cudaError_t e = ktd::launch_post_fused(ctx->post, reinterpret_cast<const float4*>(hdr), image_out,
                                                 ctx->bloom_scratch, (cudaStream_t)stream);
    if (e != cudaSuccess) return cuda_fail(e, "fused post launch");
    return KT_OK;
}

}  // extern "C"

// =========================================================================================
// CudaRenderer mirror (src/renderer/mod.rs)
// =========================================================================================
struct kt_frame {
    float* hdr = nullptr;
    uint32_t* image = nullptr;
    uint32_t* host_image = nullptr;  // pinned
    uint32_t* err = nullptr;
    uint32_t* host_err = nullptr;    // pinned, 2 words
    cudaEvent_t traced = nullptr;    // trace done (on the render stream)
    cudaEvent_t computed = nullptr;  // post done (on the post stream)
    cudaEvent_t ready = nullptr;     // image and error word in pinned memory (on the copy stream)
    bool has_event = false;
    bool used = false;               // `ready` has been recorded at least once
};

// Frames are traced on the legacy default stream (cudarc's default_stream(), like the reference),
// post-processed on a non-blocking stream of the highest priority and come back to pinned memory
// on a non-blocking copy stream.  With two frames in flight the post passes of one frame run
// while the next frame is traced: their blocks are dispatched ahead of the trace's remaining
// blocks as SMs free up, so part of their time overlaps the next trace.  The copy of one frame
// overlaps the trace of the next as well.  The post passes use the context's bloom buffer.
struct kt_renderer {
    kt_context* ctx = nullptr;
    cudaStream_t stream = nullptr;   // the legacy default stream, like cudarc's default_stream()
    cudaStream_t post = nullptr;     // non-blocking, highest priority: bloom and tone map
    cudaStream_t copy = nullptr;     // non-blocking device-to-host stream
    kt_frame frames[2];
    std::deque<uint32_t> pending;
    uint32_t next_frame = 0;
    int schedule = KT_SCHED_AUTO;
};

namespace {
void destroy_renderer(kt_renderer* r) {
    if (!r) return;
    if (r->ctx) {
        DeviceGuard g(r->ctx->device);
        cudaDeviceSynchronize();
        for (auto& f : r->frames) {
            cudaFree(f.hdr);
            cudaFree(f.image);
            cudaFree(f.err);
            cudaFreeHost(f.host_image);
            cudaFreeHost(f.host_err);
            if (f.ready) cudaEventDestroy(f.ready);
            if (f.computed) cudaEventDestroy(f.computed);
            if (f.traced) cudaEventDestroy(f.traced);
        }
        if (r->copy) cudaStreamDestroy(r->copy);
        if (r->post) cudaStreamDestroy(r->post);
        destroy_ctx(r->ctx);
    }
    delete r;
}
}  // namespace

extern "C" {

kt_status kt_renderer_new(const kt_config* cfg, int device, kt_renderer** out) {
    if (!out) return fail(KT_ERR_INVALID_ARG, "out is NULL");
    *out = nullptr;
    kt_renderer* r = new (std::nothrow) kt_renderer();
    if (!r) return fail(KT_ERR_INVALID_ARG, "out of host memory");
    kt_status st = kt_context_create(cfg, device, &r->ctx);
    if (st != KT_OK) {
        delete r;
        return st;
    }
    DeviceGuard g(device);
    const size_t px = (size_t)cfg->width * cfg->height;
    {
        int least = 0, greatest = 0;
        cudaError_t e = cudaStreamCreateWithFlags(&r->copy, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaDeviceGetStreamPriorityRange(&least, &greatest);
        if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&r->post, cudaStreamNonBlocking, greatest);
        if (e != cudaSuccess) {
            st = cuda_fail(e, "create copy and post streams");
            destroy_renderer(r);
            return st;
        }
    }
    for (auto& f : r->frames) {
        cudaError_t e;
        if ((e = cudaMalloc(&f.hdr, px * 4 * sizeof(float))) != cudaSuccess ||
            (e = cudaMalloc(&f.image, px * sizeof(uint32_t))) != cudaSuccess ||
            (e = cudaMalloc(&f.err, 2 * sizeof(uint32_t))) != cudaSuccess ||
            (e = cudaMallocHost(&f.host_image, px * sizeof(uint32_t))) != cudaSuccess ||
            (e = cudaMallocHost(&f.host_err, 2 * sizeof(uint32_t))) != cudaSuccess ||
            (e = cudaEventCreateWithFlags(&f.ready, cudaEventDisableTiming)) != cudaSuccess ||
            (e = cudaEventCreateWithFlags(&f.computed, cudaEventDisableTiming)) != cudaSuccess ||
            (e = cudaEventCreateWithFlags(&f.traced, cudaEventDisableTiming)) != cudaSuccess ||
            (e = cudaMemset(f.hdr, 0, px * 4 * sizeof(float))) != cudaSuccess ||
            (e = cudaMemset(f.image, 0, px * sizeof(uint32_t))) != cudaSuccess ||
            (e = cudaMemset(f.err, 0, 2 * sizeof(uint32_t))) != cudaSuccess) {
            st = cuda_fail(e, "allocate frame buffers");
            destroy_renderer(r);
            return st;
        }
        f.host_err[0] = f.host_err[1] = 0;
    }
    *out = r;
    return KT_OK;
}

kt_status kt_renderer_set_schedule(kt_renderer* r, int32_t schedule) {
    if (!r) return fail(KT_ERR_INVALID_ARG, "renderer is NULL");
    if (schedule < KT_SCHED_PLAIN || schedule > KT_SCHED_AUTO) return fail(KT_ERR_INVALID_ARG, "unknown schedule %d", schedule);
    r->schedule = schedule;
    return KT_OK;
}

kt_status kt_renderer_autotune(kt_renderer* r, const kt_camera* cam, uint32_t reps) {
    if (!r || !cam) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    return kt_context_autotune(r->ctx, r->stream, cam, reps, nullptr, 0, nullptr, nullptr);
}
kt_status kt_renderer_set_tuning(kt_renderer* r, const kt_tuning* tuning) {
    if (!r) return fail(KT_ERR_INVALID_ARG, "renderer is NULL");
    return kt_context_set_tuning(r->ctx, tuning);
}

kt_status kt_renderer_submit_render(kt_renderer* r, const float cam_pos[3], const float fwd[3],
                                    const float rgt[3], const float up[3], float fov_scale,
                                    int32_t* submitted) {
    if (!r || !cam_pos || !fwd || !rgt || !up) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    if (submitted) *submitted = 0;
    if (r->pending.size() == 2) return KT_OK;
    uint32_t idx = 2;
    for (uint32_t off = 0; off < 2; ++off) {
        const uint32_t cand = (r->next_frame + off) % 2;
        bool busy = false;
        for (uint32_t p : r->pending) busy = busy || p == cand;
        if (!busy) {
            idx = cand;
            break;
        }
    }
    if (idx == 2) return fail(KT_ERR_INVALID_ARG, "no free frame buffer");
    kt_frame& f = r->frames[idx];
    kt_camera cam;
    for (int i = 0; i < 3; ++i) {
        cam.cam_pos[i] = cam_pos[i];
        cam.fwd[i] = fwd[i];
        cam.rgt[i] = rgt[i];
        cam.up[i] = up[i];
    }
    cam.fov_scale = fov_scale;
    DeviceGuard g(r->ctx->device);
    const size_t px = (size_t)r->ctx->cfg.width * r->ctx->cfg.height;
    // the buffers of this frame may still be on their way to the host from its previous use
    if (f.used) KT_CUDA(cudaStreamWaitEvent(r->stream, f.ready, 0), "order after the previous copy");
    KT_CUDA(cudaMemsetAsync(f.err, 0, 2 * sizeof(uint32_t), r->stream), "clear LUT error flag");
    kt_status st = kt_trace(r->ctx, r->stream, &cam, r->schedule, f.hdr, f.err);
    if (st != KT_OK) return st;
    KT_CUDA(cudaEventRecord(f.traced, r->stream), "record trace event");
    // post passes on their own stream (one at a time: they share the context's bloom buffer)
    KT_CUDA(cudaStreamWaitEvent(r->post, f.traced, 0), "order the post passes after the trace");
    st = kt_post_fused(r->ctx, r->post, f.hdr, f.image);
    if (st != KT_OK) return st;
    KT_CUDA(cudaEventRecord(f.computed, r->post), "record render event");
    KT_CUDA(cudaStreamWaitEvent(r->copy, f.computed, 0), "order the copy after the render");
    KT_CUDA(cudaMemcpyAsync(f.host_err, f.err, 2 * sizeof(uint32_t), cudaMemcpyDeviceToHost, r->copy), "read LUT error flag");
    KT_CUDA(cudaMemcpyAsync(f.host_image, f.image, px * sizeof(uint32_t), cudaMemcpyDeviceToHost, r->copy), "copy image back");
    KT_CUDA(cudaEventRecord(f.ready, r->copy), "record frame event");
    f.used = true;
    f.has_event = true;
    r->pending.push_back(idx);
    r->next_frame = (idx + 1) % 2;
    if (submitted) *submitted = 1;
    return KT_OK;
}

kt_status kt_renderer_ready_frame(kt_renderer* r, uint32_t* index, const uint32_t** data, float* overflow_temp) {
    if (!r || !index || !data) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    if (r->pending.empty()) return KT_ERR_NOT_READY;
    const uint32_t idx = r->pending.front();
    kt_frame& f = r->frames[idx];
    if (!f.has_event) return KT_ERR_NOT_READY;
    const cudaError_t q = cudaEventQuery(f.ready);
    if (q == cudaErrorNotReady) return KT_ERR_NOT_READY;
    if (q != cudaSuccess) return cuda_fail(q, "query frame event");
    if (f.host_err[0] != 0) {
        float t;
        std::memcpy(&t, &f.host_err[1], sizeof t);
        if (overflow_temp) *overflow_temp = t;
        return fail(KT_ERR_LUT_OVERFLOW, "colour temperature above lut_max_temp: %g > %g", t, r->ctx->cfg.lut_max_temp);
    }
    *index = idx;
    *data = f.host_image;
    return KT_OK;
}

kt_status kt_renderer_finish_frame(kt_renderer* r, uint32_t index) {
    if (!r) return fail(KT_ERR_INVALID_ARG, "renderer is NULL");
    if (r->pending.empty()) return fail(KT_ERR_QUEUE_ORDER, "frame queue is empty");
    if (r->pending.front() != index)
        return fail(KT_ERR_QUEUE_ORDER, "frame queue out of order: expect=%u got=%u", r->pending.front(), index);
    r->pending.pop_front();
    r->frames[index].has_event = false;
    return KT_OK;
}

kt_status kt_renderer_wait(kt_renderer* r) {
    if (!r) return fail(KT_ERR_INVALID_ARG, "renderer is NULL");
    for (uint32_t idx : r->pending) {
        if (r->frames[idx].has_event) KT_CUDA(cudaEventSynchronize(r->frames[idx].ready), "wait for frame");
    }
    return KT_OK;
}

kt_status kt_renderer_frame_hdr(kt_renderer* r, uint32_t index, const float** hdr_dev) {
    if (!r || !hdr_dev || index > 1) return fail(KT_ERR_INVALID_ARG, "bad argument");
    *hdr_dev = r->frames[index].hdr;
    return KT_OK;
}

void kt_renderer_destroy(kt_renderer* r) { destroy_renderer(r); }

}  // extern "C"

// =========================================================================================
// Batched renders
// =========================================================================================
struct kt_batch {
    int device = 0;
    int sms = 0;
    std::vector<kt_context*> ctx;
    std::vector<kt_job> jobs;
    ktd::BatchTable* table = nullptr;
    int bx = 16, by = 16;
    int schedule = KT_SCHED_PLAIN;  // KT_SCHED_PLAIN: tiles of bx x by; KT_SCHED_WAVEFRONT: persistent units
    int blocks_per_sm = 4;          // persistent launch: resident 128-thread blocks per SM
    unsigned* counter = nullptr;    // persistent launch: the unit counter (1 word)
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaStream_t capture = nullptr;
};

namespace {
void batch_drop_graph(kt_batch* b) {
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
}
void batch_layout(kt_batch* b) {
    int tiles = 0;
    unsigned units = 0, patch_units = 0;
    for (int j = 0; j < b->table->n; ++j)
        patch_units += ktd::unit_count(b->table->job[j].sc.width, b->table->job[j].sc.height, 1, false, false);
    // warps that the GPU holds of the kernel's default shape (launch_batch_persistent)
    const unsigned warps = (unsigned)b->sms * (b->table->job[0].sc.precision == KT_PREC_FP64 ? 8u : 16u);
    for (int j = 0; j < b->table->n; ++j) {
        ktd::BatchJob& e = b->table->job[j];
        e.tiles_x = (e.sc.width + b->bx - 1) / b->bx;
        const int tiles_y = (e.sc.height + b->by - 1) / b->by;
        e.tile_begin = tiles;
        tiles += e.tiles_x * tiles_y;
        e.unit_begin = units;
        e.strips = ktd::take_strips(e.sc.width, e.sc.height, patch_units, warps) ? 1 : 0;
        units += ktd::unit_count(e.sc.width, e.sc.height, 1, false, e.strips != 0);
    }
    b->table->total_tiles = tiles;
    b->table->total_units = units;
}
cudaError_t batch_launch(kt_batch* b, cudaStream_t st) {
    if (b->schedule == KT_SCHED_WAVEFRONT) return ktd::launch_batch_persistent(*b->table, b->blocks_per_sm, b->counter, st);
    return ktd::launch_batch(*b->table, b->bx, b->by, st);
}
void batch_free(kt_batch* b) {
    if (!b) return;
    {
        DeviceGuard g(b->device);
        batch_drop_graph(b);
        if (b->capture) cudaStreamDestroy(b->capture);
        cudaFree(b->counter);
    }
    for (kt_context* c : b->ctx) destroy_ctx(c);
    delete b->table;
    delete b;
}
}  // namespace

extern "C" {

kt_status kt_batch_create(const kt_job* jobs, uint32_t n, int device, kt_batch** out) {
    if (!jobs || !out) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    *out = nullptr;
    if (n == 0 || n > KT_BATCH_MAX_JOBS)
        return fail(KT_ERR_INVALID_ARG, "a batch holds 1..%d jobs, got %u", KT_BATCH_MAX_JOBS, n);
    for (uint32_t j = 0; j < n; ++j) {
        if (!jobs[j].hdr_out || !jobs[j].err_word) return fail(KT_ERR_INVALID_ARG, "job %u: NULL output", j);
        if (jobs[j].cfg.mode != jobs[0].cfg.mode || jobs[j].cfg.precision != jobs[0].cfg.precision)
            return fail(KT_ERR_INVALID_ARG, "job %u: every job of a batch must share mode and precision", j);
    }
    kt_batch* b = new (std::nothrow) kt_batch();
    if (!b) return fail(KT_ERR_INVALID_ARG, "out of host memory");
    b->device = device;
    b->table = new (std::nothrow) ktd::BatchTable();
    if (!b->table) {
        delete b;
        return fail(KT_ERR_INVALID_ARG, "out of host memory");
    }
    b->jobs.assign(jobs, jobs + n);
    b->table->n = (int)n;
    for (uint32_t j = 0; j < n; ++j) {
        kt_context* c = nullptr;
        const kt_status st = kt_context_create(&jobs[j].cfg, device, &c);
        if (st != KT_OK) {
            batch_free(b);
            return st;
        }
        b->ctx.push_back(c);
        ktd::BatchJob& e = b->table->job[j];
        e.sc = c->scene;
        e.cam = to_camera(&jobs[j].cam);
        e.hdr = reinterpret_cast<float4*>(jobs[j].hdr_out);
        e.err = jobs[j].err_word;
    }
    {
        DeviceGuard g(device);
        cudaError_t e = cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, device);
        if (e == cudaSuccess) e = cudaMalloc(&b->counter, sizeof(unsigned));
        if (e != cudaSuccess) {
            batch_free(b);
            return cuda_fail(e, "allocate the unit counter");
        }
    }
    batch_layout(b);
    *out = b;
    return KT_OK;
}

kt_status kt_batch_set_block(kt_batch* b, int32_t bx, int32_t by) {
    if (!b) return fail(KT_ERR_INVALID_ARG, "batch is NULL");
    if (bx <= 0 || by <= 0 || (int64_t)bx * by > 1024) return fail(KT_ERR_INVALID_ARG, "block %dx%d invalid", bx, by);
    b->bx = bx;
    b->by = by;
    b->schedule = KT_SCHED_PLAIN;
    batch_layout(b);
    batch_drop_graph(b);
    return KT_OK;
}

kt_status kt_batch_set_tuning(kt_batch* b, const kt_tuning* t) {
    if (!b || !t) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    if (t->schedule == KT_SCHED_PLAIN) return kt_batch_set_block(b, t->block_x, t->block_y);
    if (t->schedule != KT_SCHED_WAVEFRONT)
        return fail(KT_ERR_INVALID_ARG, "batch tuning schedule %d must be plain or wavefront", t->schedule);
    if (t->blocks_per_sm < 4 || t->blocks_per_sm > 6)
        return fail(KT_ERR_INVALID_ARG, "batch blocks_per_sm %d not in 4..6", t->blocks_per_sm);
    b->schedule = KT_SCHED_WAVEFRONT;
    b->blocks_per_sm = t->blocks_per_sm;
    batch_drop_graph(b);
    return KT_OK;
}

kt_status kt_batch_get_tuning(const kt_batch* b, kt_tuning* t) {
    if (!b || !t) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    std::memset(t, 0, sizeof *t);
    t->schedule = b->schedule;
    t->block_x = b->schedule == KT_SCHED_PLAIN ? b->bx : 0;
    t->block_y = b->schedule == KT_SCHED_PLAIN ? b->by : 0;
    t->blocks_per_sm = b->schedule == KT_SCHED_WAVEFRONT ? b->blocks_per_sm : 4;
    t->refill_min = 1;
    return KT_OK;
}

kt_status kt_batch_set_camera(kt_batch* b, uint32_t j, const kt_camera* cam) {
    if (!b || !cam) return fail(KT_ERR_INVALID_ARG, "NULL argument");
    if ((int)j >= b->table->n) return fail(KT_ERR_INVALID_ARG, "job %u out of range", j);
    b->jobs[j].cam = *cam;
    b->table->job[j].cam = to_camera(cam);
    batch_drop_graph(b);
    return KT_OK;
}

kt_status kt_batch_trace(kt_batch* b, void* stream) {
    if (!b) return fail(KT_ERR_INVALID_ARG, "batch is NULL");
    DeviceGuard g(b->device);
    const cudaError_t e = batch_launch(b, (cudaStream_t)stream);
    if (e != cudaSuccess) return cuda_fail(e, "batch launch");
    return KT_OK;
}

kt_status kt_batch_trace_graph(kt_batch* b, void* stream) {
    if (!b) return fail(KT_ERR_INVALID_ARG, "batch is NULL");
    DeviceGuard g(b->device);
    if (!b->exec) {
        if (!b->capture) KT_CUDA(cudaStreamCreateWithFlags(&b->capture, cudaStreamNonBlocking), "create capture stream");
        KT_CUDA(cudaStreamBeginCapture(b->capture, cudaStreamCaptureModeThreadLocal), "begin capture");
        const cudaError_t le = batch_launch(b, b->capture);
        cudaGraph_t graph = nullptr;
        const cudaError_t ce = cudaStreamEndCapture(b->capture, &graph);
        if (le != cudaSuccess) {
            if (graph) cudaGraphDestroy(graph);
            return cuda_fail(le, "batch launch under capture");
        }
        if (ce != cudaSuccess) return cuda_fail(ce, "end capture");
        b->graph = graph;
        const cudaError_t ie = cudaGraphInstantiate(&b->exec, b->graph, 0);
        if (ie != cudaSuccess) {
            batch_drop_graph(b);
            return cuda_fail(ie, "instantiate graph");
        }
    }
    KT_CUDA(cudaGraphLaunch(b->exec, (cudaStream_t)stream), "launch graph");
    return KT_OK;
}

kt_status kt_batch_autotune(kt_batch* b, void* stream, uint32_t reps, kt_tune_entry* table, uint32_t* n_entries) {
    if (!b) return fail(KT_ERR_INVALID_ARG, "batch is NULL");
    if (reps == 0 || reps > 64) return fail(KT_ERR_INVALID_ARG, "kt_batch_autotune: reps must be in 1..64");
    DeviceGuard g(b->device);
    cudaStream_t st = (cudaStream_t)stream;
    kt_tuning saved;
    kt_batch_get_tuning(b, &saved);
    std::vector<kt_tuning> cands;
    static const int kPlain[][2] = {{16, 16}, {32, 8}, {8, 8}, {16, 8}, {8, 16}, {32, 4}};
    for (const auto& s2 : kPlain) {
        kt_tuning t{};
        t.schedule = KT_SCHED_PLAIN;
        t.block_x = s2[0];
        t.block_y = s2[1];
        t.blocks_per_sm = 4;
        t.refill_min = 1;
        cands.push_back(t);
    }
    const bool variants = b->jobs[0].cfg.precision == KT_PREC_FP32 && b->jobs[0].cfg.mode == KT_MODE_REF;
    for (int bps = 4; bps <= (variants ? 6 : 4); ++bps) {
        kt_tuning t{};
        t.schedule = KT_SCHED_WAVEFRONT;
        t.blocks_per_sm = bps;
        t.refill_min = 1;
        cands.push_back(t);
    }
    // first candidate's images of every job, kept for the bit-identity test of the others
    size_t total = 0;
    for (const kt_job& j : b->jobs) total += (size_t)j.cfg.width * j.cfg.height;
    float4* keep = nullptr;
    unsigned long long* diff = nullptr;
    std::vector<cudaEvent_t> ev(2 * reps, nullptr);
    auto release = [&]() {
        cudaFree(keep);
        cudaFree(diff);
        for (cudaEvent_t e : ev)
            if (e) cudaEventDestroy(e);
    };
    cudaError_t e;
    if ((e = cudaMalloc(&keep, total * sizeof(float4))) != cudaSuccess ||
        (e = cudaMalloc(&diff, sizeof(unsigned long long))) != cudaSuccess) {
        release();
        return cuda_fail(e, "kt_batch_autotune: allocate scratch");
    }
    for (cudaEvent_t& x : ev)
        if ((e = cudaEventCreate(&x)) != cudaSuccess) {
            release();
            return cuda_fail(e, "kt_batch_autotune: create events");
        }
    std::vector<kt_tune_entry> rows;
    kt_status out = KT_OK;
    for (size_t i = 0; i < cands.size() && out == KT_OK; ++i) {
        if ((out = kt_batch_set_tuning(b, &cands[i])) != KT_OK) break;
        if ((e = batch_launch(b, st)) != cudaSuccess) { out = cuda_fail(e, "kt_batch_autotune: launch"); break; }
        unsigned long long mism = 0;
        size_t off = 0;
        for (const kt_job& j : b->jobs) {
            const size_t n = (size_t)j.cfg.width * j.cfg.height;
            if (i == 0) {
                e = cudaMemcpyAsync(keep + off, j.hdr_out, n * sizeof(float4), cudaMemcpyDeviceToDevice, st);
            } else {
                unsigned long long d = 0;
                if ((e = ktd::launch_count_mismatch(j.hdr_out, keep + off, n, diff, st)) == cudaSuccess)
                    e = cudaMemcpyAsync(&d, diff, sizeof d, cudaMemcpyDeviceToHost, st);
                mism += d;
            }
            if (e != cudaSuccess) break;
            off += n;
        }
        if (e != cudaSuccess) { out = cuda_fail(e, "kt_batch_autotune: compare images"); break; }
        for (uint32_t r = 0; r < reps && e == cudaSuccess; ++r) {
            if ((e = cudaEventRecord(ev[2 * r], st)) == cudaSuccess && (e = batch_launch(b, st)) == cudaSuccess)
                e = cudaEventRecord(ev[2 * r + 1], st);
        }
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) { out = cuda_fail(e, "kt_batch_autotune: timed launches"); break; }
        std::vector<float> ms(reps);
        for (uint32_t r = 0; r < reps; ++r) cudaEventElapsedTime(&ms[r], ev[2 * r], ev[2 * r + 1]);
        std::sort(ms.begin(), ms.end());
        kt_tune_entry row;
        row.tuning = cands[i];
        row.ms = ms[reps / 2];
        row.identical = mism == 0 ? 1 : 0;
        rows.push_back(row);
    }
    release();
    if (out != KT_OK) {
        kt_batch_set_tuning(b, &saved);
        return out;
    }
    size_t best = 0;
    for (size_t i = 1; i < rows.size(); ++i)
        if (rows[i].identical && rows[i].ms < rows[best].ms) best = i;
    if ((out = kt_batch_set_tuning(b, &rows[best].tuning)) != KT_OK) return out;
    if (table)
        for (size_t i = 0; i < rows.size(); ++i) table[i] = rows[i];
    if (n_entries) *n_entries = (uint32_t)rows.size();
    return KT_OK;
}

kt_status kt_batch_trace_sequential(kt_batch* b, void* stream, int32_t schedule) {
    if (!b) return fail(KT_ERR_INVALID_ARG, "batch is NULL");
    for (size_t j = 0; j < b->ctx.size(); ++j) {
        const kt_status st = kt_trace(b->ctx[j], stream, &b->jobs[j].cam, schedule, b->jobs[j].hdr_out, b->jobs[j].err_word);
        if (st != KT_OK) return st;
    }
    return KT_OK;
}

uint64_t kt_batch_rays(const kt_batch* b) {
    if (!b) return 0;
    uint64_t r = 0;
    for (const kt_job& j : b->jobs) r += (uint64_t)j.cfg.width * j.cfg.height * j.cfg.spp;
    return r;
}

void kt_batch_destroy(kt_batch* b) { batch_free(b); }

}  // extern "C"

