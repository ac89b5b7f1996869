// tonemap.cu -- linear HDR image -> RGBA8 on the GPU: exposure (optionally automatic), the
// reference's per-pixel colour chain, tone curve and sRGB quantisation.
//
// The chain restates render::render's per-pixel loop (src/render.rs:3100-3260) for its
// colour steps, with the tone curves and gamma_correct of src/render.rs:3608-3658 and the
// auto-exposure key value of src/render.rs:2594-2606 (log-average luminance,
// src/render.rs:525-540).  The colour steps run in f64 like the reference's; the tone curve and
// sRGB power run in f32 with an f64 re-evaluation near byte boundaries (tone_gamma), so the
// bytes agree with an f64 restatement except where a last-bit difference meets a boundary.
//
// Kernels (HBM-bound: 12 bytes in, 4 bytes out per pixel):
//   k_loglum   fixed grid of 256 x 256 threads, each summing ln(1e-4 + max(lum, 0)) (f32 log,
//              f64 sum) over a grid stride, a shared-memory tree per block -> 256 partials.  The
//              grid does not depend on the device, so the sum is reproducible.
//   k_tonemap  4 pixels per thread: three 16-byte loads of 12 floats, one 16-byte store of
//              4 RGBA pixels (a scalar tail with byte stores for pixel counts not divisible
//              by 4, or for buffers that are not 16-byte aligned).  With auto-exposure each block first
//              sums the 256 partials in the same fixed order.  Dithered chains, unaligned buffers and
//              tone curves whose table does not fit take the f32 path with its f64 fallback.
//   k_tonemap_graded  chains with the other optional steps on 16-byte aligned buffers: colour steps
//              in f64, byte tables for the rest.
//   k_tonemap_flat  the common chain (no optional step) on 16-byte aligned buffers: each channel's
//              byte from a table of the chain's 255 byte thresholds (one entry lookup per
//              channel, see ByteTable).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>

#include "../../include/luminara_gpu.h"
#include "kernels.h"
#include "scene_access.h"
#include "table_cache.h"

namespace lum {
namespace tone {

constexpr int kLogBlocks = 256;
constexpr int kLogThreads = 256;
constexpr int kLogAhead = 8;          // steps of k_loglum whose loads are in flight together
constexpr int kThreads = 256;
static_assert(kLogBlocks * sizeof(double) <= LUM_TONEMAP_SCRATCH_BYTES, "scratch too small");

struct Chain {
    lum_tonemap_params p;
    double cos_h, sin_h;          // hue rotation
    int16_t bright_off;           // (brightness * 255) as i16
    bool wb, hue, sat, grade, bright, contrast, sepia, tint, balance;
    bool extra;                   // any step beyond exposure, tone curve and gamma
    float inv_gamma;              // 1/gamma, or 0 for the sRGB transfer function
    double wb_r, wb_g, wb_b;      // white-balance factors
    double hue_d, hue_m, hue_p;   // hue rotation matrix (a circulant)
};

// Rust's `as u8` from f64: truncation, saturating, NaN -> 0.
__host__ __device__ __forceinline__ uint32_t sat_u8(double x) {
    if (!(x > 0.0)) return 0u;
    if (x >= 255.0) return 255u;
    return (uint32_t)x;
}

__host__ __device__ __forceinline__ double clamp01(double x) { return fmin(fmax(x, 0.0), 1.0); }

// Tone curves (src/render.rs:3608-3641).
__host__ __device__ __forceinline__ double tone_curve(int kind, double x) {
    x = fmax(x, 0.0);   // f64::max ignores NaN
    switch (kind) {
        case LUM_TONEMAP_REINHARD:
            return x / (1.0 + x);
        case LUM_TONEMAP_FILMIC: {
            auto uc2 = [](double v) {
                const double a = 0.15, b = 0.50, c = 0.10, d = 0.20, e = 0.02, f = 0.30;
                return ((v * (a * v + c * b) + d * e) / (v * (a * v + b) + d * f)) - e / f;
            };
            return clamp01(uc2(x) / uc2(11.2));
        }
        case LUM_TONEMAP_NONE:
            return clamp01(x);
        default: {
            const double a = 2.51, b = 0.03, c = 2.43, d = 0.59, e = 0.14;
            return clamp01((x * (a * x + b)) / (x * (c * x + d) + e));
        }
    }
}

// Tone curve in f32 (the fast path of tone_gamma below).
__device__ __forceinline__ float tone_curve_f(int kind, float x) {
    x = fmaxf(x, 0.0f);
    switch (kind) {
        case LUM_TONEMAP_REINHARD:
            return x / (1.0f + x);
        case LUM_TONEMAP_FILMIC: {
            auto uc2 = [](float v) {
                const float a = 0.15f, b = 0.50f, c = 0.10f, d = 0.20f, e = 0.02f, f = 0.30f;
                return ((v * (a * v + c * b) + d * e) / (v * (a * v + b) + d * f)) - e / f;
            };
            return fminf(fmaxf(uc2(x) / uc2(11.2f), 0.0f), 1.0f);
        }
        case LUM_TONEMAP_NONE:
            return fminf(fmaxf(x, 0.0f), 1.0f);
        default: {
            const float a = 2.51f, b = 0.03f, c = 2.43f, d = 0.59f, e = 0.14f;
            return fminf(fmaxf((x * (a * x + b)) / (x * (c * x + d) + e), 0.0f), 1.0f);
        }
    }
}

// gamma_correct (src/render.rs:3648-3658): sRGB transfer function (gamma <= 0) or 1/gamma
// power, plus the dither offset, quantised as (s + dither).clamp(0, 0.999) * 256.
__host__ __device__ __forceinline__ double quantised(double s, double dither) {
    double q = s + dither;
    if (q != q) return -1.0;
    return fmin(fmax(q, 0.0), 0.999) * 256.0;
}

__host__ __device__ __forceinline__ double srgb64(double x, double gamma) {
    if (gamma > 0.0) return pow(x, 1.0 / gamma);
    return x <= 0.0031308 ? 12.92 * x : 1.055 * pow(x, 1.0 / 2.4) - 0.055;
}

// Tone curve + gamma_correct of one channel.  The tone curve and the power run in f32: from an
// exact f64 input their result moves the scaled value q by less than 1e-4 of a byte step.  Only
// when q lies within 1e-3 of an integer, where truncation could then differ from the f64
// result, is the channel evaluated again in f64; so the bytes are those of the f64 formulas at
// a fraction of their cost.
__device__ __noinline__ double tone_gamma64(int kind, double x, double gamma, double dither) {
    return quantised(srgb64(clamp01(tone_curve(kind, x)), gamma), dither);
}

__device__ __forceinline__ uint32_t tone_gamma(int kind, double x, double gamma, double dither) {
    if (x != x) return 0u;
    const float t = tone_curve_f(kind, (float)x);
    float sf;
    if (gamma > 0.0) sf = powf(t, (float)(1.0 / gamma));
    else sf = t <= 0.0031308f ? 12.92f * t : 1.055f * powf(t, 1.0f / 2.4f) - 0.055f;
    double q = quantised((double)sf, dither);
    const double fr = q - floor(q);
    if (fr < 2e-3 || fr > 1.0 - 2e-3) q = tone_gamma64(kind, x, gamma, dither);
    return q < 0.0 ? 0u : sat_u8(q);
}

// a / b for a finite a and b = 1, 2, ... with r = 1 / b: the quotient corrected by its exact remainder
// (Markstein, IBM J. Res. Dev. 1990).  No difference from the division in 2^30 draws with b up to 2^27; a
// proof would need the first quotient within one ulp, and its two roundings give 1.5.
__device__ __forceinline__ double quotient(double a, double b, double r) {
    const double q = a * r;
    return fma(fma(-q, b, a), r, q);
}

// White balance, hue, saturation and grading of one pixel (src/render.rs:3120-3180).
__device__ __forceinline__ void colour_steps(const Chain& C, double& cr, double& cg, double& cb) {
    const lum_tonemap_params& P = C.p;
    if (C.wb) {
        cr *= C.wb_r;
        cb *= C.wb_b;
        cg *= C.wb_g;
    }
    if (C.hue) {   // rotation about the grey axis (Rodrigues)
        const double d = C.hue_d, m = C.hue_m, p = C.hue_p;
        const double nr = cr * d + cg * m + cb * p;
        const double ng = cr * p + cg * d + cb * m;
        const double nb = cr * m + cg * p + cb * d;
        cr = fmax(nr, 0.0);
        cg = fmax(ng, 0.0);
        cb = fmax(nb, 0.0);
    }
    if (C.sat) {
        const double lum = 0.2126 * cr + 0.7152 * cg + 0.0722 * cb;
        cr = lum + (cr - lum) * P.saturation;
        cg = lum + (cg - lum) * P.saturation;
        cb = lum + (cb - lum) * P.saturation;
    }
    if (C.grade) {
        const double lum = fmax(0.2126 * cr + 0.7152 * cg + 0.0722 * cb, 0.0);
        const double t = clamp01(lum / (lum + 1.0));
        cr *= P.grade_shadows[0] * (1.0 - t) + P.grade_highlights[0] * t;
        cg *= P.grade_shadows[1] * (1.0 - t) + P.grade_highlights[1] * t;
        cb *= P.grade_shadows[2] * (1.0 - t) + P.grade_highlights[2] * t;
    }
}

// The steps on quantised bytes (src/render.rs:3200-3260): brightness and contrast, then sepia across
// the channels, then tint, colour balance and posterise.
__device__ __forceinline__ uint32_t byte_before(const Chain& C, uint32_t v) {
    if (C.bright) v = (uint32_t)min(max((int)v + (int)C.bright_off, 0), 255);
    if (C.contrast) v = sat_u8(fmin(fmax((((double)v / 255.0 - 0.5) * C.p.contrast + 0.5) * 255.0, 0.0), 255.0));
    return v;
}
__device__ __forceinline__ void sepia(double s, uint32_t& R, uint32_t& G, uint32_t& B) {
    const double fr = R / 255.0, fg = G / 255.0, fb = B / 255.0;
    const double sr = fmin(fr * 0.393 + fg * 0.769 + fb * 0.189, 1.0);
    const double sg = fmin(fr * 0.349 + fg * 0.686 + fb * 0.168, 1.0);
    const double sb = fmin(fr * 0.272 + fg * 0.534 + fb * 0.131, 1.0);
    R = sat_u8((fr * (1.0 - s) + sr * s) * 255.0);
    G = sat_u8((fg * (1.0 - s) + sg * s) * 255.0);
    B = sat_u8((fb * (1.0 - s) + sb * s) * 255.0);
}
__device__ __forceinline__ uint32_t byte_after(const Chain& C, int c, uint32_t v) {
    const lum_tonemap_params& P = C.p;
    if (C.tint) v = sat_u8(fmin(fmax((v / 255.0 * P.tint[c]) * 255.0, 0.0), 255.0));
    if (C.balance) v = sat_u8(fmin(fmax(v * P.color_balance[c], 0.0), 255.0));
    if (P.posterize >= 2) {
        const double L = (double)P.posterize;
        v = sat_u8(fmin(fmax(round((v / 255.0) * (L - 1.0)) / (L - 1.0) * 255.0, 0.0), 255.0));
    }
    return v;
}

// One pixel of the full chain (src/render.rs:3100-3260); pixel p = j * w + i of the output.
__device__ __noinline__ uint32_t pixel_full(const Chain& C, double r, double g, double b, uint32_t p, uint32_t w,
                                            uint32_t h, double exposure) {
    const lum_tonemap_params& P = C.p;
    uint32_t i = 0, j = 0;
    if (P.vignette > 0.0 || P.dither) {
        j = p / w;
        i = p - j * w;
    }
    double vf = 1.0;
    if (P.vignette > 0.0) {
        const double cx = ((double)i + 0.5) / (double)w - 0.5, cy = ((double)j + 0.5) / (double)h - 0.5;
        vf = fmax(1.0 - (cx * cx + cy * cy) * P.vignette * 4.0, 0.0);
    }
    double cr = r * exposure * vf, cg = g * exposure * vf, cb = b * exposure * vf;
    colour_steps(C, cr, cg, cb);
    double dither = 0.0;
    if (P.dither) {   // 4x4 Bayer matrix (src/render.rs:3187-3195), (value - 0.5) / 255
        const uint64_t bayer = 0x5D7F91B36E4CA280ull;   // rows {0,8,2,10} {12,4,14,6} {3,11,1,9} {15,7,13,5}
        const uint32_t v = (uint32_t)(bayer >> (4 * ((j & 3) * 4 + (i & 3)))) & 15u;
        dither = ((double)v / 16.0 - 0.5) / 255.0;
    }
    uint32_t R = tone_gamma(P.tone_map, cr, P.gamma, dither), G = tone_gamma(P.tone_map, cg, P.gamma, dither),
             B = tone_gamma(P.tone_map, cb, P.gamma, dither);
    R = byte_before(C, R);
    G = byte_before(C, G);
    B = byte_before(C, B);
    if (C.sepia) sepia(P.sepia, R, G, B);
    R = byte_after(C, 0, R);
    G = byte_after(C, 1, G);
    B = byte_after(C, 2, B);
    return R | (G << 8) | (B << 16) | (255u << 24);
}

// Fast channel path: tone curve KIND and the sRGB / 1/gamma power in f32 with the hardware
// reciprocal and __powf (exp2 of log2), then the exact f64 evaluation (tone_gamma64) only when
// the scaled value lies within kGuard of a byte boundary.  Values below one step are byte 0
// either way.
template <int KIND>
__device__ __forceinline__ float tone_fast(float x) {
    x = fmaxf(x, 0.0f);
    if constexpr (KIND == LUM_TONEMAP_REINHARD) {
        return __fdividef(x, 1.0f + x);
    } else if constexpr (KIND == LUM_TONEMAP_FILMIC) {
        auto uc2 = [](float v) {
            const float a = 0.15f, b = 0.50f, c = 0.10f, d = 0.20f, e = 0.02f, f = 0.30f;
            return __fdividef(fmaf(v, fmaf(a, v, c * b), d * e), fmaf(v, fmaf(a, v, b), d * f)) - e / f;
        };
        const float white = 1.0f / uc2(11.2f);
        return fminf(fmaxf(uc2(x) * white, 0.0f), 1.0f);
    } else if constexpr (KIND == LUM_TONEMAP_NONE) {
        return fminf(x, 1.0f);
    } else {
        const float a = 2.51f, b = 0.03f, c = 2.43f, d = 0.59f, e = 0.14f;
        return fminf(fmaxf(__fdividef(x * fmaf(a, x, b), fmaf(x, fmaf(c, x, d), e)), 0.0f), 1.0f);
    }
}

// Guard window, in byte steps, around each quantisation boundary.  Worst case of the f32 path:
// 1 ulp for the exposure product, 2 ulp __fdividef, 6 ulp __powf (2 + floor(1.173 |y log2 t|)
// with y = 1/2.4 and t >= 0.0031308), a few ulp of fmaf/scaling: < 1.1e-6 relative, i.e. at most
// 2.7e-4 of a step at the top of the range.  The window keeps a 2x margin over that.
constexpr float kGuard = 6e-4f;

// v: the channel before exposure; the exact f64 input of the fallback is (double)v * exposure.
template <int KIND>
__device__ __forceinline__ uint32_t tone_gamma_fast(float v, float exposure32, double exposure, float inv_gamma) {
    const float x = v * exposure32;
    if (x != x) return 0u;
    const float t = tone_fast<KIND>(x);
    float sv;
    if (inv_gamma > 0.0f) sv = __powf(t, inv_gamma);
    else sv = t <= 0.0031308f ? 12.92f * t : fmaf(1.055f, __powf(t, 1.0f / 2.4f), -0.055f);
    const float q = fminf(fmaxf(sv, 0.0f), 0.999f) * 256.0f;
    const float fr = q - floorf(q);
    if (fr > 1.0f - kGuard || (fr < kGuard && q >= 1.0f)) {
        const double q64 = tone_gamma64(KIND, (double)v * exposure, inv_gamma > 0.0f ? 1.0 / (double)inv_gamma : 0.0,
                                        0.0);
        return q64 < 0.0 ? 0u : sat_u8(q64);
    }
    return (uint32_t)q;
}

// Byte tables of the common chain.  Without dither, vignette or the other optional steps, a
// channel's byte is a non-decreasing step function of x = (double)v * exposure: the tone curve,
// the sRGB or 1/gamma power and the quantisation are all monotone.  So it is fixed by the 255
// thresholds T_k = min{x : byte(x) >= k}, found once per (tone curve, gamma) on the host by
// bisection over the f64 bit patterns with the reference's own f64 formulas (the host's libm
// pow, as the f64 restatement uses) -- exact, not a fit.  The kernel finds x's byte from one
// table entry: positive doubles order like their bit patterns, and the bucket of x is its top
// 19 bits (sign, exponent, 7 mantissa bits), chosen so that no bucket holds two thresholds.
// Entry i (a u64): byte at the bucket's lower end in bits 56-63, the low 45 bits of the bucket's
// threshold (or 2^45: none) in bits 0-45; x's byte is that base, plus one if x's low 45 bits reach
// the threshold's.  Entry 0 stands for every bucket below the first, entry nb + 1 for every
// bucket above the last.  Non-finite, huge or non-positive x take the f64 path as before.
constexpr int kTabShift = 45;                                  // 52 - 7 mantissa bits
constexpr unsigned long long kTabLowMask = (1ull << kTabShift) - 1ull;
constexpr int kTabMaxEntries = 4096;                           // nb + 2 per table

struct ByteTable {
    const unsigned long long* tab;   // device address of the slot, or null: no table
    const uint32_t* tab32;           // the same entries for f32 keys (k_tonemap_flat)
    long long k0;                    // bucket key of entry 1
    int nb;                          // buckets with an entry of their own
};
constexpr int kTabSlots = TableCache<ByteTable>::kSlots;       // (tone curve, gamma) pairs per device

static __device__ __align__(256) unsigned long long g_byte_tables[kTabSlots][kTabMaxEntries];
// 32-bit entries for a power-of-two exposure, where x's bits below the bucket are the low 16 bits m
// of v followed by 29 zeros: byte << 16 plus 2^16 - ceil(threshold / 2^29), so that adding m carries
// into the byte exactly when m reaches the threshold.
static __device__ __align__(256) uint32_t g_byte_tables32[kTabSlots][kTabMaxEntries];

template <int KIND>
__device__ __forceinline__ uint32_t tone_table(float v, double exposure, const ByteTable& T, float inv_gamma) {
    const double x = (double)v * exposure;
    if (!(x > 0.0)) return 0u;                                 // NaN, zero and negatives: byte 0
    if (!(x < 1e30)) {
        const double q64 = tone_gamma64(KIND, x, inv_gamma > 0.0f ? 1.0 / (double)inv_gamma : 0.0, 0.0);
        return q64 < 0.0 ? 0u : sat_u8(q64);
    }
    const long long b = __double_as_longlong(x);
    const long long i = min(max((b >> kTabShift) - T.k0 + 1, 0ll), (long long)T.nb + 1);
    const unsigned long long e = __ldg(T.tab + i);
    return (uint32_t)(e >> 56) + (((unsigned long long)b & kTabLowMask) >= (e & (2ull * kTabLowMask + 1ull)) ? 1u : 0u);
}

template <int KIND>
__device__ __forceinline__ uint32_t pixel_table(float r, float g, float b, double exposure, const ByteTable& T,
                                                float inv_gamma) {
    const uint32_t R = tone_table<KIND>(r, exposure, T, inv_gamma);
    const uint32_t G = tone_table<KIND>(g, exposure, T, inv_gamma);
    const uint32_t B = tone_table<KIND>(b, exposure, T, inv_gamma);
    return R | (G << 8) | (B << 16) | (255u << 24);
}

// The common chain -- exposure, tone curve KIND, sRGB or gamma -- inline, in f32 with the exact
// f64 fallback near byte boundaries (the channel values stay f32 until the fallback needs them);
// used when no byte table is available.
template <int KIND>
__device__ __forceinline__ uint32_t pixel_fast(float r, float g, float b, float e32, double exposure, float inv_gamma) {
    const uint32_t R = tone_gamma_fast<KIND>(r, e32, exposure, inv_gamma);
    const uint32_t G = tone_gamma_fast<KIND>(g, e32, exposure, inv_gamma);
    const uint32_t B = tone_gamma_fast<KIND>(b, e32, exposure, inv_gamma);
    return R | (G << 8) | (B << 16) | (255u << 24);
}

// Any chain: the fast path, or pixel_full (kept out of line so the hot loop stays small in the
// instruction cache) when an optional step is on.
template <int KIND>
__device__ __forceinline__ uint32_t pixel_rgba(const Chain& C, float r, float g, float b, uint32_t p, uint32_t w,
                                               uint32_t h, float e32, double exposure) {
    if (C.extra) return pixel_full(C, r, g, b, p, w, h, exposure);
    return pixel_fast<KIND>(r, g, b, e32, exposure, C.inv_gamma);
}

__device__ __forceinline__ double log_lum(float r, float g, float b) {
    const double lum = 0.2126 * (double)r + 0.7152 * (double)g + 0.0722 * (double)b;
    return (double)logf((float)(1e-4 + fmax(lum, 0.0)));   // f32 log, f64 sum
}

// VEC: 4 pixels per step from three 16-byte loads (hdr 16-byte aligned).
template <bool VEC>
__global__ void __launch_bounds__(kLogThreads) k_loglum(const float* __restrict__ hdr, uint32_t n, double* __restrict__ partials) {
    __shared__ double sh[kLogThreads];
    double acc = 0.0;
    const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    uint32_t from = 0;
    if constexpr (VEC) {
        const float4* in = reinterpret_cast<const float4*>(hdr);
        const uint32_t n4 = n / 4;
        // kLogAhead steps' loads at once (the 256 blocks leave a third of the SMs one block each, so
        // a step's latency counts): 4K with auto-exposure, 1 / 2 / 4 / 8 steps 67.5 / 64.3 / 61.6 /
        // 60.7 us.  The sums stay in the order of one step after another.
        for (uint64_t q = t0; q < n4; q += (uint64_t)kLogAhead * stride) {
            float4 f[kLogAhead][3];
#pragma unroll
            for (int k = 0; k < kLogAhead; ++k) {
                const uint64_t p = q + (uint64_t)k * stride;
                if (p < n4)
                    for (int j = 0; j < 3; ++j) f[k][j] = in[3 * p + j];
            }
#pragma unroll
            for (int k = 0; k < kLogAhead; ++k) {
                const float4 a = f[k][0], b = f[k][1], c = f[k][2];
                if (q + (uint64_t)k * stride < n4)
                    acc += (log_lum(a.x, a.y, a.z) + log_lum(a.w, b.x, b.y)) + (log_lum(b.z, b.w, c.x) + log_lum(c.y, c.z, c.w));
            }
        }
        from = 4 * n4;
    }
    for (uint32_t p = from + t0; p < n; p += stride)
        acc += log_lum(hdr[3 * (size_t)p], hdr[3 * (size_t)p + 1], hdr[3 * (size_t)p + 2]);
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int s = kLogThreads / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) partials[blockIdx.x] = sh[0];
}

template <bool VEC, int KIND>
__global__ void __launch_bounds__(kThreads, 6) k_tonemap(const float* __restrict__ hdr, uint32_t w, uint32_t h, const __grid_constant__ Chain C,
                                                      double exposure, const double* __restrict__ partials,
                                                      uint8_t* __restrict__ rgba, const ByteTable T) {
    __shared__ double s_exposure;
    if (partials) {   // auto-exposure: key value 0.18 over the log-average luminance
        if (threadIdx.x == 0) {
            double sum = 0.0;
            for (int k = 0; k < kLogBlocks; ++k) sum += partials[k];
            const size_t n = (size_t)w * h;
            const double log_avg = n ? exp(sum / (double)n) : 0.0;
            s_exposure = (log_avg > 1e-6 ? 0.18 / log_avg : 1.0) * exposure;
        }
        __syncthreads();
        exposure = s_exposure;
    }
    const uint32_t n = w * h;
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x;
    const float e32 = (float)exposure;
    uint32_t scalar_from = 0;
    if constexpr (VEC) {
        const uint32_t n4 = n / 4;
        const float4* in = reinterpret_cast<const float4*>(hdr);
        uint4* out = reinterpret_cast<uint4*>(rgba);
        if (!C.extra && T.tab) {   // the common chain from its byte table, exposures the flat kernel leaves out (uniform branch, hoisted)
            const float ig = C.inv_gamma;
            for (uint32_t q = t0; q < n4; q += stride) {
                const float4 a = __ldcs(in + 3 * q), b = __ldcs(in + 3 * q + 1), c = __ldcs(in + 3 * q + 2);
                __stcs(out + q, make_uint4(pixel_table<KIND>(a.x, a.y, a.z, exposure, T, ig),
                                           pixel_table<KIND>(a.w, b.x, b.y, exposure, T, ig),
                                           pixel_table<KIND>(b.z, b.w, c.x, exposure, T, ig),
                                           pixel_table<KIND>(c.y, c.z, c.w, exposure, T, ig)));
            }
        } else if (!C.extra) {     // the common chain in f32 with the exact fallback
            const float ig = C.inv_gamma;
            for (uint32_t q = t0; q < n4; q += stride) {
                const float4 a = __ldcs(in + 3 * q), b = __ldcs(in + 3 * q + 1), c = __ldcs(in + 3 * q + 2);
                __stcs(out + q, make_uint4(pixel_fast<KIND>(a.x, a.y, a.z, e32, exposure, ig),
                                           pixel_fast<KIND>(a.w, b.x, b.y, e32, exposure, ig),
                                           pixel_fast<KIND>(b.z, b.w, c.x, e32, exposure, ig),
                                           pixel_fast<KIND>(c.y, c.z, c.w, e32, exposure, ig)));
            }
        } else {
            for (uint32_t q = t0; q < n4; q += stride) {
                const float4 a = in[3 * q], b = in[3 * q + 1], c = in[3 * q + 2];
                const uint32_t p = 4 * q;
                out[q] = make_uint4(pixel_rgba<KIND>(C, a.x, a.y, a.z, p, w, h, e32, exposure),
                                    pixel_rgba<KIND>(C, a.w, b.x, b.y, p + 1, w, h, e32, exposure),
                                    pixel_rgba<KIND>(C, b.z, b.w, c.x, p + 2, w, h, e32, exposure),
                                    pixel_rgba<KIND>(C, c.y, c.z, c.w, p + 3, w, h, e32, exposure));
            }
        }
        scalar_from = 4 * n4;
    }
    for (uint32_t p = scalar_from + t0; p < n; p += stride) {   // any output alignment: byte stores
        const uint32_t v = pixel_rgba<KIND>(C, hdr[3 * (size_t)p], hdr[3 * (size_t)p + 1], hdr[3 * (size_t)p + 2], p,
                                            w, h, e32, exposure);
        rgba[4 * (size_t)p] = (uint8_t)v;
        rgba[4 * (size_t)p + 1] = (uint8_t)(v >> 8);
        rgba[4 * (size_t)p + 2] = (uint8_t)(v >> 16);
        rgba[4 * (size_t)p + 3] = (uint8_t)(v >> 24);
    }
}

// Exposure with auto-exposure: key value 0.18 over the log-average luminance, the partials summed in
// their fixed order (the loads by all threads, the sum by one).  Called by the whole block.
__device__ __forceinline__ double auto_exposure(const double* __restrict__ partials, size_t n, double exposure) {
    __shared__ double s_part[kLogBlocks];
    __shared__ double s_exposure;
    for (int k = threadIdx.x; k < kLogBlocks; k += blockDim.x) s_part[k] = partials[k];
    __syncthreads();
    if (threadIdx.x == 0) {
        double sum = 0.0;
#pragma unroll 8
        for (int k = 0; k < kLogBlocks; ++k) sum += s_part[k];
        const double log_avg = n ? exp(sum / (double)n) : 0.0;
        s_exposure = (log_avg > 1e-6 ? 0.18 / log_avg : 1.0) * exposure;
    }
    __syncthreads();
    return s_exposure;
}

// Four channels through tone_table, out of line: the flat kernel's rare values (|v| >= 2^97, infinite
// or NaN) and its last n % 4 pixels.
template <int KIND>
__device__ __noinline__ uint32_t word_table(float4 q, double exposure, const unsigned long long* tab, long long k0, int nb,
                                            float inv_gamma) {
    const ByteTable T{tab, nullptr, k0, nb};
    return tone_table<KIND>(q.x, exposure, T, inv_gamma) | (tone_table<KIND>(q.y, exposure, T, inv_gamma) << 8) |
           (tone_table<KIND>(q.z, exposure, T, inv_gamma) << 16) | (tone_table<KIND>(q.w, exposure, T, inv_gamma) << 24);
}

// The common chain from its byte table.  A channel's byte depends on that channel alone, so the
// image is a flat run of floats: a warp takes 128 pixels as 96 float4 in lane order (each load
// 512 consecutive bytes), turns each float4 into four bytes, and regroups those three bytes per
// pixel through 384 bytes of shared memory.  The table sits in shared memory, with 4-byte entries
// for a power-of-two exposure (POW2: `off` takes v's top 16 bits to an entry; the low 16 added to it
// carry into the byte at the threshold), 8-byte ones otherwise.  Four blocks of 256 threads per SM
// with one tile's loads ahead.  Bound by HBM: 8K frame (531 MB) 88 us, 6.03 TB/s, 0.92 of the
// measured copy rate; the table read through L1 by one pixel quad per thread was bound by the L1's
// wavefronts (80% of its peak; 48-byte lane strides and 8-byte gathers) and took 131 us.  1080p
// 14.4 -> 11.3 us, 4K with auto-exposure 83 -> 66 us.  Without the loads ahead 92-95 us at 4-6
// blocks/SM; 3 or 5 blocks with them 95-97 us.
constexpr int kFlatThreads = 256;
constexpr int kFlatBlocks = 4;
// Exposures 2^-k..2^k that the flat kernel takes: within them every finite v keeps x in the range where
// the table stands for the f64 formulas (below 2^117 above the last threshold, and denormal v far
// below the first); others take k_tonemap's tables.
constexpr int kFlatExposureLog2 = 20;

template <int KIND, bool POW2>
__global__ void __launch_bounds__(kFlatThreads, kFlatBlocks) k_tonemap_flat(const float* __restrict__ hdr, uint32_t n, int off,
                                                                   double exposure, const double* __restrict__ partials,
                                                                   uint8_t* __restrict__ rgba, const ByteTable T,
                                                                   float inv_gamma) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ uint32_t s_pack[kFlatThreads / 32][96];
    auto* t32 = reinterpret_cast<uint32_t*>(s_raw);
    auto* t64 = reinterpret_cast<unsigned long long*>(s_raw);
    const int top = T.nb + 1;
    for (int i = threadIdx.x; i <= top; i += kFlatThreads) {
        if constexpr (POW2) t32[i] = __ldg(T.tab32 + i);
        else t64[i] = __ldg(T.tab + i);
    }
    if (partials) exposure = auto_exposure(partials, n, exposure);
    __syncthreads();
    auto byte_of = [&](float v) -> uint32_t {
        if constexpr (POW2) {
            const int u = __float_as_int(v);
            return (t32[min(max((u >> 16) + off, 0), top)] + ((uint32_t)u & 0xFFFFu)) >> 16;
        } else {
            const double x = (double)v * exposure;
            const long long b = __double_as_longlong(x);
            const int hi = (int)(b >> 32);
            const unsigned long long e = t64[min(max((hi >> (kTabShift - 32)) - (int)T.k0 + 1, 0), top)];
            return (uint32_t)(e >> 56) + (((unsigned long long)b & kTabLowMask) >= (e & (2ull * kTabLowMask + 1ull)) ? 1u : 0u);
        }
    };
    const int lane = threadIdx.x & 31;
    uint32_t* pack = s_pack[threadIdx.x >> 5];
    const uint32_t n4 = n / 4, lim = 3 * n4, chunks = (n4 + 31) / 32;
    const float4* in = reinterpret_cast<const float4*>(hdr);
    uint4* out = reinterpret_cast<uint4*>(rgba);
    const uint32_t step = gridDim.x * (kFlatThreads / 32);
    float4 f[3];
    auto fetch = [&](uint32_t c) {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const uint32_t i = 96 * c + 32 * j + lane;
            f[j] = c < chunks && i < lim ? __ldcs(in + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    uint32_t c = blockIdx.x * (kFlatThreads / 32) + (threadIdx.x >> 5);
    fetch(c);
    for (; c < chunks; c += step) {
        const float4 cur[3] = {f[0], f[1], f[2]};
        if (c < chunks - min(chunks, step)) fetch(c + step);   // the next tile's loads fly meanwhile
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const float4 q = cur[j];
            uint32_t w = byte_of(q.x) | (byte_of(q.y) << 8) | (byte_of(q.z) << 16) | (byte_of(q.w) << 24);
            const uint32_t m = max(max(__float_as_uint(q.x) << 1, __float_as_uint(q.y) << 1),
                                   max(__float_as_uint(q.z) << 1, __float_as_uint(q.w) << 1));
            if (m >= 0xE0000000u)   // |v| >= 2^97
                w = word_table<KIND>(q, exposure, T.tab, T.k0, T.nb, inv_gamma);
            pack[32 * j + lane] = w;
        }
        __syncwarp();
        const uint32_t w0 = pack[3 * lane], w1 = pack[3 * lane + 1], w2 = pack[3 * lane + 2];
        const uint32_t g = 32 * c + lane;
        if (g < n4)
            __stcs(out + g, make_uint4((w0 & 0xFFFFFFu) | 0xFF000000u, (w0 >> 24) | ((w1 & 0xFFFFu) << 8) | 0xFF000000u,
                                       (w1 >> 16) | ((w2 & 0xFFu) << 16) | 0xFF000000u, (w2 >> 8) | 0xFF000000u));
        __syncwarp();
    }
    if (blockIdx.x == 0 && threadIdx.x < n - 4 * n4) {
        const float* v = hdr + 3 * (size_t)(4 * n4 + threadIdx.x);
        reinterpret_cast<uint32_t*>(rgba)[4 * n4 + threadIdx.x] =
            word_table<KIND>(make_float4(v[0], v[1], v[2], 0.0f), exposure, T.tab, T.k0, T.nb, inv_gamma) | 0xFF000000u;
    }
}

// Chains with optional steps other than dither: one pixel per lane and tile of 32, its colour steps
// in f64 as in pixel_full, each channel's byte from the byte table (shared memory), the steps on
// bytes from tables of the 256 bytes that each block fills first.  pixel_full evaluated the curve and
// the power per channel and six divisions per pixel, and was bound by instruction fetch (5.6 stalled
// warps per issue): 1080p with auto-exposure, grading, vignette and contrast 140 -> 40 us with
// k_loglum (25 MB twice: 8 us at the copy rate; the f64 steps bound it now).  3 / 4 / 5 / 6 blocks/SM
// 39.9 / 41.0 / 43.1 / 43.1 us.
constexpr int kGradedThreads = 256;
constexpr int kGradedBlocks = 3;
template <int KIND>
__global__ void __launch_bounds__(kGradedThreads, kGradedBlocks)
    k_tonemap_graded(const float* __restrict__ hdr, uint32_t w, uint32_t h, const __grid_constant__ Chain C, double exposure,
                     const double* __restrict__ partials, uint8_t* __restrict__ rgba, const ByteTable T) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ uint8_t s_before[256], s_after[3][256];
    __shared__ float4 s_px[kGradedThreads / 32][24];   // written so, read as 96 floats
    static_assert(alignof(decltype(s_px)) == 16, "the stores are 16 bytes wide");
    auto* tab = reinterpret_cast<unsigned long long*>(s_raw);
    const int top = T.nb + 1;
    for (int i = threadIdx.x; i <= top; i += kGradedThreads) tab[i] = __ldg(T.tab + i);
    static_assert(kGradedThreads == 256, "one byte per thread");
    s_before[threadIdx.x] = (uint8_t)byte_before(C, threadIdx.x);
    for (int c = 0; c < 3; ++c) s_after[c][threadIdx.x] = (uint8_t)byte_after(C, c, threadIdx.x);
    const uint32_t n = w * h;
    if (partials) exposure = auto_exposure(partials, n, exposure);
    __syncthreads();
    const lum_tonemap_params& P = C.p;
    auto byte_of = [&](double x) -> uint32_t {
        if (!(x < 1e30)) {   // NaN (byte 0) and x beyond the table's range
            const double q64 = x != x ? -1.0 : tone_gamma64(KIND, x, P.gamma, 0.0);
            return q64 < 0.0 ? 0u : sat_u8(q64);
        }
        const long long b = __double_as_longlong(x);   // zero and negatives come before entry 1: byte 0
        const unsigned long long e = tab[min(max((int)(b >> kTabShift) - (int)T.k0 + 1, 0), top)];
        return (uint32_t)(e >> 56) + (((unsigned long long)b & kTabLowMask) >= (e & (2ull * kTabLowMask + 1ull)) ? 1u : 0u);
    };
    const int lane = threadIdx.x & 31;
    const float* px = reinterpret_cast<const float*>(s_px[threadIdx.x >> 5]);
    const double dw = (double)w, dh = (double)h, rw = 1.0 / dw, rh = 1.0 / dh;
    const uint32_t tiles = (n + 31) / 32, step = gridDim.x * (kGradedThreads / 32), lim = 3 * (n / 4);
    const float4* in = reinterpret_cast<const float4*>(hdr);
    auto fetch = [&](uint32_t t) {
        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t >= tiles || lane >= 24) return f;
        const uint32_t i = 24 * t + lane;
        if (i < lim) return __ldcs(in + i);
        const uint64_t k = 4 * (uint64_t)i, end = 3 * (uint64_t)n;   // the last n % 4 pixels
        if (k < end) f.x = hdr[k];
        if (k + 1 < end) f.y = hdr[k + 1];
        if (k + 2 < end) f.z = hdr[k + 2];
        if (k + 3 < end) f.w = hdr[k + 3];
        return f;
    };
    uint32_t t = blockIdx.x * (kGradedThreads / 32) + (threadIdx.x >> 5);
    float4 f = fetch(t);
    for (; t < tiles; t += step) {
        if (lane < 24) s_px[threadIdx.x >> 5][lane] = f;
        if (t < tiles - min(tiles, step)) f = fetch(t + step);
        __syncwarp();
        const double r = px[3 * lane], g = px[3 * lane + 1], b = px[3 * lane + 2];
        __syncwarp();
        const uint32_t p = 32 * t + lane;
        double cr = r * exposure, cg = g * exposure, cb = b * exposure;
        if (P.vignette > 0.0) {
            const uint32_t j = p / w, i = p - j * w;
            const double cx = quotient((double)i + 0.5, dw, rw) - 0.5, cy = quotient((double)j + 0.5, dh, rh) - 0.5;
            const double vf = fmax(1.0 - (cx * cx + cy * cy) * P.vignette * 4.0, 0.0);
            cr *= vf;
            cg *= vf;
            cb *= vf;
        }
        colour_steps(C, cr, cg, cb);
        uint32_t R = s_before[byte_of(cr)], G = s_before[byte_of(cg)], B = s_before[byte_of(cb)];
        if (C.sepia) sepia(P.sepia, R, G, B);
        if (p < n)
            __stcs(reinterpret_cast<uint32_t*>(rgba) + p,
                   s_after[0][R] | ((uint32_t)s_after[1][G] << 8) | ((uint32_t)s_after[2][B] << 16) | 0xFF000000u);
    }
}

Chain make_chain(const lum_tonemap_params& p) {
    Chain C;
    C.p = p;
    const double ang = p.hue_shift * (3.14159265358979323846 / 180.0);
    C.cos_h = std::cos(ang);
    C.sin_h = std::sin(ang);
    {
        const double k = 1.0 / 3.0, s3 = 1.0 / std::sqrt(3.0), ca = C.cos_h, sa = C.sin_h;
        C.hue_d = ca + k * (1.0 - ca);
        C.hue_m = k * (1.0 - ca) - s3 * sa;
        C.hue_p = k * (1.0 - ca) + s3 * sa;
    }
    C.wb_r = 1.0 + p.white_balance * 0.1;
    C.wb_g = 1.0 + p.white_balance * 0.02;
    C.wb_b = 1.0 - p.white_balance * 0.1;
    double bo = p.brightness * 255.0;
    bo = bo != bo ? 0.0 : (bo > 32767.0 ? 32767.0 : (bo < -32768.0 ? -32768.0 : bo));
    C.bright_off = (int16_t)bo;
    auto ne1 = [](const double* v) { return v[0] != 1.0 || v[1] != 1.0 || v[2] != 1.0; };
    C.wb = std::fabs(p.white_balance) > 1e-6;
    C.hue = std::fabs(p.hue_shift) > 1e-6;
    C.sat = std::fabs(p.saturation - 1.0) > 1e-6;
    C.grade = ne1(p.grade_shadows) || ne1(p.grade_highlights);
    C.bright = std::fabs(p.brightness) > 1e-6;
    C.contrast = std::fabs(p.contrast - 1.0) > 1e-6;
    C.sepia = p.sepia > 0.0;
    C.tint = p.tint[0] < 1.0 || p.tint[1] < 1.0 || p.tint[2] < 1.0;
    C.balance = std::fabs(p.color_balance[0] - 1.0) > 1e-6 || std::fabs(p.color_balance[1] - 1.0) > 1e-6 ||
                std::fabs(p.color_balance[2] - 1.0) > 1e-6;
    C.inv_gamma = p.gamma > 0.0 ? (float)(1.0 / p.gamma) : 0.0f;
    C.extra = p.vignette > 0.0 || p.dither || p.posterize >= 2 || C.wb || C.hue || C.sat || C.grade || C.bright ||
              C.contrast || C.sepia || C.tint || C.balance;
    return C;
}

// Host side of the byte tables: the chain's byte for an exact f64 x (gamma <= 0: sRGB).
static uint32_t host_byte(int kind, double x, double gamma) {
    return sat_u8(quantised(srgb64(clamp01(tone_curve(kind, x)), gamma), 0.0));
}

static long long dbits(double x) {
    long long b;
    std::memcpy(&b, &x, sizeof b);
    return b;
}
static double bdouble(long long b) {
    double x;
    std::memcpy(&x, &b, sizeof x);
    return x;
}

// Builds the entries of one table; false when the chain is not the step function the table
// encodes (a bucket with two thresholds, too many buckets, or a byte that does not match).
static bool build_byte_table(int kind, double gamma, std::vector<unsigned long long>& ent, long long& k0, int& nb) {
    const long long top = dbits(1e30);
    std::vector<long long> th;                                  // bit patterns of T_1 .. T_bmax
    const uint32_t bmax = host_byte(kind, 1e30, gamma);
    if (host_byte(kind, bdouble(1), gamma) != 0u) return false;  // smallest positive x must be byte 0
    for (uint32_t k = 1; k <= bmax; ++k) {
        long long lo = th.empty() ? 0 : th.back() - 1, hi = top;   // byte(lo) < k <= byte(hi)
        if (lo < 0) lo = 0;
        while (hi - lo > 1) {
            const long long m = lo + (hi - lo) / 2;
            if (host_byte(kind, bdouble(m), gamma) >= k) hi = m;
            else lo = m;
        }
        th.push_back(hi);
    }
    if (th.empty()) return false;
    k0 = th.front() >> kTabShift;
    const long long k1 = th.back() >> kTabShift;
    nb = (int)(k1 - k0 + 1);
    if (nb + 2 > kTabMaxEntries) return false;
    ent.assign(nb + 2, 0ull);
    ent[0] = 2ull * kTabLowMask + 1ull;                          // below: byte 0, no threshold
    ent[nb + 1] = ((unsigned long long)bmax << 56) | (2ull * kTabLowMask + 1ull);
    size_t t = 0;                                               // thresholds at or below the bucket start
    for (int i = 0; i < nb; ++i) {
        const long long key = k0 + i, lo = key << kTabShift, hi = (key + 1) << kTabShift;
        while (t < th.size() && th[t] <= lo) ++t;
        const uint32_t base = (uint32_t)t;
        if (host_byte(kind, bdouble(lo), gamma) != base) return false;        // not monotone here
        unsigned long long thr = 2ull * kTabLowMask + 1ull;     // none
        if (t < th.size() && th[t] < hi) {
            if (t + 1 < th.size() && th[t + 1] < hi) return false;            // two in one bucket
            thr = (unsigned long long)th[t] & kTabLowMask;
        }
        ent[i + 1] = ((unsigned long long)base << 56) | thr;
    }
    return true;
}

// Copies a table into its slot, on a stream of its own and with this thread's capture mode relaxed: a copy
// on the default stream would break a stream capture of this thread or, in the global mode, of any.
template <class T>
static bool upload_table(T (&symbol)[kTabSlots][kTabMaxEntries], const std::vector<T>& ent, int slot, void** base) {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) return false;
    cudaStream_t stream = nullptr;
    bool ok = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking) == cudaSuccess;
    if (ok) {
        ok = cudaGetSymbolAddress(base, symbol) == cudaSuccess &&
             cudaMemcpyAsync(static_cast<T*>(*base) + (size_t)slot * kTabMaxEntries, ent.data(), ent.size() * sizeof(T),
                             cudaMemcpyHostToDevice, stream) == cudaSuccess;
        ok = cudaStreamSynchronize(stream) == cudaSuccess && ok;
        cudaStreamDestroy(stream);
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
    return ok;
}

// One table per (device, tone curve, gamma), uploaded once into a slot of g_byte_tables.  graded: for a
// chain with optional steps.
static ByteTable byte_table(int kind, double gamma, bool graded) {
    static std::mutex mu;
    static TableCache<ByteTable> cache;
    const ByteTable none{nullptr, nullptr, 0, 0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return none;
    if (!(gamma > 0.0)) gamma = 0.0;
    const long long gb = dbits(gamma);
    std::lock_guard<std::mutex> lk(mu);
    bool known = false;
    if (const ByteTable* t = cache.find(dev, kind, gb, &known)) return *t;
    const int slot = cache.free_slot(dev, graded);
    if (known || slot < 0) return none;
    ByteTable T = none;
    std::vector<unsigned long long> ent;
    std::vector<uint32_t> ent32;
    if (!build_byte_table(kind, gamma, ent, T.k0, T.nb)) {
        cache.add_failed(dev, kind, gb);
        return none;
    }
    for (const unsigned long long e : ent) {
        const unsigned long long thr = e & (2ull * kTabLowMask + 1ull);
        const uint32_t t16 = thr > kTabLowMask ? 65536u : (uint32_t)((thr + (1ull << 29) - 1) >> 29);
        ent32.push_back(((uint32_t)(e >> 56) << 16) + 65536u - t16);
    }
    void *base = nullptr, *base32 = nullptr;
    if (!upload_table(g_byte_tables, ent, slot, &base) || !upload_table(g_byte_tables32, ent32, slot, &base32)) {
        cudaGetLastError();                                     // the next call tries again
        return none;
    }
    T.tab = static_cast<const unsigned long long*>(base) + (size_t)slot * kTabMaxEntries;
    T.tab32 = static_cast<const uint32_t*>(base32) + (size_t)slot * kTabMaxEntries;
    cache.add(dev, kind, gb, slot, T);
    return T;
}

}  // namespace tone

cudaError_t launch_tonemap(const float* hdr, uint32_t w, uint32_t h, const lum_tonemap_params& tm, double exposure,
                           double* scratch, uint8_t* rgba, cudaStream_t stream) {
    const size_t n = (size_t)w * h;
    if (n == 0) return cudaSuccess;
    if (n >= ((size_t)1 << 32)) return cudaErrorInvalidValue;   // 32-bit pixel indices
    const double* partials = nullptr;
    const bool vec = (((uintptr_t)hdr | (uintptr_t)rgba) & 15) == 0;
    if (tm.auto_exposure) {
        if (((uintptr_t)hdr & 15) == 0)
            tone::k_loglum<true><<<tone::kLogBlocks, tone::kLogThreads, 0, stream>>>(hdr, (uint32_t)n, scratch);
        else
            tone::k_loglum<false><<<tone::kLogBlocks, tone::kLogThreads, 0, stream>>>(hdr, (uint32_t)n, scratch);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        partials = scratch;
    }
    const tone::Chain C = tone::make_chain(tm);
    const tone::ByteTable T = C.extra ? tone::ByteTable{nullptr, nullptr, 0, 0} : tone::byte_table(tm.tone_map, tm.gamma, false);
    tone::ByteTable G{nullptr, nullptr, 0, 0};   // of the graded kernel
    if (C.extra && !tm.dither && vec) G = tone::byte_table(tm.tone_map, tm.gamma, true);
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const size_t work = vec ? (n + 3) / 4 : n;
    // at most two resident waves (6 blocks/SM), threads looping over the rest: on B200 the 1080p
    // frame 20.5 -> 18.4 us against one block per 256 quads (2.3 waves), the 8K frame unchanged
    const int grid = (int)std::min<size_t>((work + tone::kThreads - 1) / tone::kThreads, (size_t)nsm * 12);
    long long eb;
    std::memcpy(&eb, &exposure, sizeof eb);
    const int k2 = (int)((eb >> 52) & 0x7FF) - 1023;
    const bool fits = exposure > 0.0 && k2 >= -tone::kFlatExposureLog2 && k2 < tone::kFlatExposureLog2;
    const bool pow2 = fits && !partials && (eb & 0xFFFFFFFFFFFFFll) == 0;
    auto go = [&](auto kind) {
        constexpr int K = decltype(kind)::value;
        if (vec && !C.extra && T.tab && fits) {
            const size_t warps = (n / 4 + 31) / 32;
            const int fg = (int)std::max<size_t>(1, std::min<size_t>((warps + 7) / 8, (size_t)nsm * tone::kFlatBlocks));
            const int off = ((k2 + 896) << 7) - (int)T.k0 + 1;
            const size_t ents = (size_t)T.nb + 2;
            if (pow2)
                tone::k_tonemap_flat<K, true><<<fg, tone::kFlatThreads, 4 * ents, stream>>>(hdr, (uint32_t)n, off, exposure, partials,
                                                                                           rgba, T, C.inv_gamma);
            else
                tone::k_tonemap_flat<K, false><<<fg, tone::kFlatThreads, 8 * ents, stream>>>(hdr, (uint32_t)n, 0, exposure, partials,
                                                                                            rgba, T, C.inv_gamma);
            return;
        }
        if (vec && C.extra && !tm.dither && G.tab) {
            const size_t warps = (n + 31) / 32;
            const int gg = (int)std::max<size_t>(1, std::min<size_t>((warps + 7) / 8, (size_t)nsm * tone::kGradedBlocks));
            tone::k_tonemap_graded<K><<<gg, tone::kGradedThreads, 8 * ((size_t)G.nb + 2), stream>>>(
                hdr, (uint32_t)w, (uint32_t)h, C, exposure, partials, rgba, G);
            return;
        }
        if (vec)
            tone::k_tonemap<true, K><<<grid, tone::kThreads, 0, stream>>>(hdr, (uint32_t)w, (uint32_t)h, C, exposure,
                                                                          partials, rgba, T);
        else
            tone::k_tonemap<false, K><<<grid, tone::kThreads, 0, stream>>>(hdr, (uint32_t)w, (uint32_t)h, C, exposure,
                                                                           partials, rgba, T);
    };
    switch (tm.tone_map) {
        case LUM_TONEMAP_REINHARD: go(std::integral_constant<int, LUM_TONEMAP_REINHARD>()); break;
        case LUM_TONEMAP_FILMIC: go(std::integral_constant<int, LUM_TONEMAP_FILMIC>()); break;
        case LUM_TONEMAP_NONE: go(std::integral_constant<int, LUM_TONEMAP_NONE>()); break;
        default: go(std::integral_constant<int, LUM_TONEMAP_ACES>()); break;
    }
    return cudaGetLastError();
}

}  // namespace lum

extern "C" {

void lum_tonemap_default(lum_tonemap_params* out) {
    if (!out) return;
    std::memset(out, 0, sizeof *out);
    out->tone_map = LUM_TONEMAP_ACES;                                   // src/render.rs:176-182
    out->exposure = 1.0;
    out->gamma = 0.0;
    out->saturation = 1.0;
    out->contrast = 1.0;
    for (int c = 0; c < 3; ++c) {
        out->grade_shadows[c] = out->grade_highlights[c] = 1.0;
        out->tint[c] = out->color_balance[c] = 1.0;
    }
}

lum_status lum_tonemap_device(const float* d_hdr_rgb, uint32_t width, uint32_t height, const lum_tonemap_params* tm,
                              void* d_scratch, uint8_t* d_rgba, void* stream) {
    if (!tm) return lum::set_error(LUM_ERR_INVALID_ARGUMENT, "null tone-map parameters");
    if ((size_t)width * height == 0) return LUM_OK;
    if ((size_t)width * height >= ((size_t)1 << 32))
        return lum::set_error(LUM_ERR_TOO_LARGE, "tone map supports fewer than 2^32 pixels");
    if (!d_hdr_rgb || !d_rgba) return lum::set_error(LUM_ERR_INVALID_ARGUMENT, "null image buffer");
    if ((uintptr_t)d_hdr_rgb & 3u) return lum::set_error(LUM_ERR_INVALID_ARGUMENT, "d_hdr_rgb is not 4-byte aligned");
    if (d_scratch && ((uintptr_t)d_scratch & 7u))
        return lum::set_error(LUM_ERR_INVALID_ARGUMENT, "d_scratch is not 8-byte aligned");
    if (tm->auto_exposure && !d_scratch)
        return lum::set_error(LUM_ERR_INVALID_ARGUMENT, "auto_exposure needs LUM_TONEMAP_SCRATCH_BYTES of device scratch");
    if (tm->tone_map < LUM_TONEMAP_ACES || tm->tone_map > LUM_TONEMAP_NONE)
        return lum::set_error(LUM_ERR_INVALID_ARGUMENT, "unknown tone_map");
    cudaError_t e = lum::launch_tonemap(d_hdr_rgb, width, height, *tm, tm->exposure, (double*)d_scratch, d_rgba,
                                        (cudaStream_t)stream);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return lum::set_error(LUM_ERR_CUDA, cudaGetErrorString(e));
    }
    return LUM_OK;
}

}  // extern "C"
