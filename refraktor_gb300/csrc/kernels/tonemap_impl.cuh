// Tonemap kernel body shared by two translation units: image.cu compiles it
// with full-precision math (PRECISE) and tonemap_fast.cu with -use_fast_math,
// the way the reference builds assets/kernels/tonemap.cu
// (src/librefrakt/src/image/tonemapper.cpp:10-22), so that the fast variant
// matches the reference kernel.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>

#include "image_kernels.h"

namespace rfk_tm {
// ----------------------------------------------------------------- tonemap --
template <int C, bool HALF>
struct pixel_out;
template <>
struct pixel_out<3, true> {
    static __device__ void store(void* out, size_t i, float r, float g, float b, float) {
        __half* o = reinterpret_cast<__half*>(out) + 3 * i;
        o[0] = __float2half_rn(r);
        o[1] = __float2half_rn(g);
        o[2] = __float2half_rn(b);
    }
};
template <>
struct pixel_out<4, true> {
    static __device__ void store(void* out, size_t i, float r, float g, float b, float a) {
        __half2 lo = __floats2half2_rn(r, g), hi = __floats2half2_rn(b, a);
        uint2 v;
        v.x = *reinterpret_cast<unsigned*>(&lo);
        v.y = *reinterpret_cast<unsigned*>(&hi);
        reinterpret_cast<uint2*>(out)[i] = v;
    }
};
template <>
struct pixel_out<3, false> {
    static __device__ void store(void* out, size_t i, float r, float g, float b, float) {
        float* o = reinterpret_cast<float*>(out) + 3 * i;
        o[0] = r;
        o[1] = g;
        o[2] = b;
    }
};
template <>
struct pixel_out<4, false> {
    static __device__ void store(void* out, size_t i, float r, float g, float b, float a) {
        reinterpret_cast<float4*>(out)[i] = make_float4(r, g, b, a);
    }
};

__device__ __forceinline__ float sat(float v) { return fminf(fmaxf(v, 0.0f), 1.0f); }
__device__ __forceinline__ float lerpf(float a, float b, float t) { return a + t * (b - a); }

// flam3-style highlight handling (an extension; the reference parses
// highlight_power but never applies it): when the brightest channel of the
// density-scaled colour exceeds 1, scale it to 1 and reduce saturation by
// (1/max)^highlight_power so that hot pixels go white instead of shifting hue.
__device__ void highlight(float& r, float& g, float& b, float hp) {
    const float m = fmaxf(r, fmaxf(g, b));
    if (!(m > 1.0f)) return;
    const float s = 1.0f / m;
    const float ratio = powf(s, hp);
    // at HSV value 1 a channel is 1 - sat * k(hue); scaling sat by `ratio`
    // maps each channel c to 1 - ratio * (1 - c)
    r = 1.0f - ratio * (1.0f - r * s);
    g = 1.0f - ratio * (1.0f - g * s);
    b = 1.0f - ratio * (1.0f - b * s);
}

// The block's part of a density histogram (density_histo.cu:1-42, granularity
// 4: 97 log2 bins, max density): 32-bit counts in shared memory (a block sees
// fewer than 2^32 pixels), the largest density as the bits of a float >= 1
// (positive floats order as their bits).
struct density_counts {
    unsigned bins[RFK_HISTOGRAM_BINS];
    unsigned max_bits;
    __device__ void clear() {
        for (int i = threadIdx.x; i < RFK_HISTOGRAM_BINS; i += blockDim.x) bins[i] = 0;
        if (threadIdx.x == 0) max_bits = 0;
        __syncthreads();
    }
    __device__ static unsigned bin(float v, float log_div) {
        if (!(v >= 1.0f)) return 0;
        const unsigned long long b = (unsigned long long)(logf(v) * log_div) + 1;
        return b >= RFK_HISTOGRAM_BINS ? RFK_HISTOGRAM_BINS - 1 : (unsigned)b;
    }
    // every thread, after its last pixel, with the largest density it saw (0: none >= 1)
    __device__ void flush(float my_max, unsigned long long* hist, unsigned long long* max_density) {
        const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(my_max));
        if ((threadIdx.x & 31) == 0 && m) atomicMax(&max_bits, m);
        __syncthreads();
        for (int i = threadIdx.x; i < RFK_HISTOGRAM_BINS; i += blockDim.x)
            if (bins[i]) atomicAdd(&hist[i], (unsigned long long)bins[i]);
        if (threadIdx.x == 0 && max_bits) atomicMax(max_density, (unsigned long long)__uint_as_float(max_bits));
    }
};

#ifdef RFK_TONEMAP_FAST
// w^(1/gamma) / w as a pair of floats. The reference evaluates w^(1/gamma) in
// FP64, which this part runs at 1/64 of the FP32 rate (a 1366 x 768 image with its
// density histogram 70-91 us that way, 19 us now); in pairs of FP32 numbers the factor is within 2^-34.8
// of it (20 M densities 2^-60 .. 2^40, gamma 1 .. 5), so that a channel times it
// rounds to the same float but for 3 in 100000, one ulp off.
//   w = 2^e m, m in [sqrt(1/2), sqrt(2)): ln m = 2 atanh(s), s = (m - 1) / (m + 1),
//   by its power series; y = (1/gamma - 1) log2 w = n + j / 32 + f; 2^y = 2^n
//   2^(j / 32) e^(f ln 2) with the table's 2^(j / 32) and a quartic in f ln 2.
// Products that an addition follows are __fmul_rn, which is not contracted.
struct pow_table {
    float2 t[32];  // 2^(j / 32) as a pair
    float2 q;      // 1 / gamma - 1 as a pair
};
__device__ __forceinline__ bool pow_pair(float w, const float2* __restrict__ table, float2 q, float& hi, float& lo) {
    const unsigned u = __float_as_uint(w);
    if (u - 0x00800000u >= 0x7f800000u - 0x00800000u) return false;  // negative, zero, subnormal, infinite, NaN
    const int e = (int)(u - 0x3f3504f3u) >> 23;
    const float m = __uint_as_float(u - ((unsigned)e << 23));
    const float num = m - 1.0f, dh = m + 1.0f, dl = m - (dh - 1.0f);
    const float sh = __fdividef(num, dh);
    const float sl = __fdividef(fmaf(-sh, dl, fmaf(-sh, dh, num)), dh);
    const float s2h = __fmul_rn(sh, sh), s2l = fmaf(2.0f * sh, sl, fmaf(sh, sh, -s2h));
    float p = fmaf(1.0f / 15, s2h, 1.0f / 13);
    p = fmaf(p, s2h, 1.0f / 11);
    p = fmaf(p, s2h, 1.0f / 9);
    p = fmaf(p, s2h, 1.0f / 7);
    p = fmaf(p, s2h, 0.2f);
    const float third = (float)(1.0 / 3), third_l = (float)(1.0 / 3 - (double)third);
    const float c = __fmul_rn(s2h, p), ch = third + c, cl = (c - (ch - third)) + third_l;
    const float uh = __fmul_rn(s2h, ch), ul = fmaf(s2l, ch, fmaf(s2h, cl, fmaf(s2h, ch, -uh)));
    const float vh = 1.0f + uh, vl = (uh - (vh - 1.0f)) + ul;
    const float lh = __fmul_rn(sh, vh), ll = fmaf(sl, vh, fmaf(sh, vl, fmaf(sh, vh, -lh)));
    constexpr double k2 = 2.8853900817779268147;  // 2 / ln 2
    const float kh = (float)k2, kl = (float)(k2 - (double)kh);
    const float gh = __fmul_rn(lh, kh), gl = fmaf(ll, kh, fmaf(lh, kl, fmaf(lh, kh, -gh)));
    const float ef = (float)e, th = ef + gh, tl = (gh - (th - ef)) + gl;
    const float yh = __fmul_rn(th, q.x), yl = fmaf(tl, q.x, fmaf(th, q.y, fmaf(th, q.x, -yh)));
    if (!(fabsf(yh) < 120.0f)) return false;
    const int n = __float2int_rn(yh * 32.0f);
    const float f = fmaf((float)n, -1.0f / 32, yh), g = f + yl, fl = yl - (g - f);
    constexpr double l2 = 0.69314718055994530942;
    const float l2h = (float)l2, l2l = (float)(l2 - (double)l2h);
    const float rh = __fmul_rn(g, l2h), rl = fmaf(fl, l2h, fmaf(g, l2l, fmaf(g, l2h, -rh)));
    const float r2 = fmaf(__fmul_rn(rh, rh), fmaf(rh, fmaf(rh, 1.0f / 24, 1.0f / 6), 0.5f), rl);
    const float2 t = table[n & 31];
    const float ph = __fmul_rn(t.x, rh), pl = fmaf(t.x, r2, fmaf(t.x, rh, -ph)) + fmaf(t.y, rh, t.y);
    const float z = t.x + ph, zl = (ph - (z - t.x)) + pl;
    const float scale = __uint_as_float((unsigned)(127 + (n >> 5)) << 23);
    hi = z * scale;
    lo = zl * scale;
    return true;
}
// col * (hi + lo), rounded once up to the pair's own error
__device__ __forceinline__ float mul_pair(float col, float hi, float lo) {
    const float p = __fmul_rn(col, hi);
    return p + fmaf(col, lo, fmaf(col, hi, -p));
}
#endif

// Per pixel (assets/kernels/tonemap.cu:67-104 with the host constant of
// src/librefrakt/src/image/tonemapper.cpp:52):
//   w = density, k2 = 10^(-log10(q) - 0.5)
//   f = 0.5 * brightness * log10(1 + w k2) / w;  (r, g, b, w) *= f
//   z = w^(1/gamma) (FP64), gf = z / w
//   c = sat(lerp(c^(1/gamma), c gf, vibrancy))
//   alpha = sat(ln(w_in) * (4 / ln 2) / 96)
// The precise build uses log1pf / powf / logf at full precision; the fast
// build is the same text under -use_fast_math, as the reference kernel. The
// density histogram of density_histo.cu:1-42
// (granularity 4: 97 log2 bins, max density) is accumulated in the same pass
// when `hist` is non-null.
// Bound by memory once a pixel costs about 100 instructions: with vibrancy 1
// and gamma >= 1 (the usual genome) the precise build leaves out the three
// c^(1/gamma) whose weight is 0, and the next pixel's load is in flight while
// this one is computed. 1920 x 1080 half4 at vibrancy 1: 12.5 us a call, 17.1-18.7
// with all four powf.
#ifdef RFK_TONEMAP_FAST
constexpr int kBlocksPerSm = 4;  // the FP64 fallback holds 62 registers
#else
constexpr int kBlocksPerSm = 6;
#endif
template <int C, bool HALF>
__global__ void __launch_bounds__(256, kBlocksPerSm) tonemap_kernel(const float4* __restrict__ bins, void* __restrict__ out, unsigned size,
                                                      float gamma, float scale_constant, float brightness, float vibrancy,
                                                      float highlight_power, unsigned long long* __restrict__ hist,
                                                      unsigned long long* __restrict__ max_density,
                                                      const unsigned long long* __restrict__ q_hits, double q_per_hit
#ifdef RFK_TONEMAP_FAST
                                                      , const __grid_constant__ pow_table pt
#endif
) {
    __shared__ density_counts counts;
    if (hist) counts.clear();
#ifdef RFK_TONEMAP_FAST
    __shared__ float2 table[32];
    if (threadIdx.x < 32) table[threadIdx.x] = pt.t[threadIdx.x];
    __syncthreads();
#endif
    if (q_hits) {
        // quality from a device counter (batched renders): the host constant
        // of the single-image path, computed here in single precision
        const float q = (float)((double)*q_hits * q_per_hit);
        scale_constant = powf(10.0f, -log10f(q) - 0.5f);
    }
    const float log_div = 4.0f / logf(2.0f);
    const double inv_gamma = 1.0 / (double)gamma;
    const float inv_gamma_f = (float)inv_gamma;
#ifndef RFK_TONEMAP_FAST
    const bool full_vibrancy = vibrancy == 1.0f && gamma >= 1.0f;
#endif
    float my_max = 0.0f;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    float4 next = i < size ? bins[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (; i < size; i += stride) {
        float4 col = next;
        if (i + stride < size) next = bins[i + stride];
        if (hist) {
            atomicAdd(&counts.bins[density_counts::bin(col.w, log_div)], 1u);
            if (col.w >= 1.0f) my_max = fmaxf(my_max, col.w);
        }
        if (col.w == 0.0f) {
            pixel_out<C, HALF>::store(out, i, 0.0f, 0.0f, 0.0f, 0.0f);
            continue;
        }
        const float input_density = col.w;
#ifdef RFK_TONEMAP_FAST
        float lg = logf(1.0f + col.w * scale_constant);
#else
        float lg = log1pf(col.w * scale_constant);
#endif
        const float factor = 0.5f * brightness * lg * 0.434294481903251827651128918916f / col.w;
        col.x *= factor;
        col.y *= factor;
        col.z *= factor;
        col.w *= factor;
        float lr, lgc, lb;
#ifdef RFK_TONEMAP_FAST
        float hi, lo;
        if (pow_pair(col.w, table, pt.q, hi, lo)) {
            lr = mul_pair(col.x, hi, lo);
            lgc = mul_pair(col.y, hi, lo);
            lb = mul_pair(col.z, hi, lo);
        } else {
            // the reference's FP64 w^(1/gamma) / w
            const double gamma_factor = pow((double)col.w, inv_gamma) / col.w;
            lr = (float)(col.x * gamma_factor);
            lgc = (float)(col.y * gamma_factor);
            lb = (float)(col.z * gamma_factor);
        }
#else
        // w^(1/gamma) / w = w^(1/gamma - 1) in one FP32 powf (2 ulp): FP64 pow
        // is slow on this part and the result is already within 1e-6 relative
        const float gamma_factor = powf(col.w, inv_gamma_f - 1.0f);
        lr = col.x * gamma_factor;
        lgc = col.y * gamma_factor;
        lb = col.z * gamma_factor;
#endif
        if (highlight_power >= 0.0f) highlight(lr, lgc, lb, highlight_power);
#ifndef RFK_TONEMAP_FAST
        if (full_vibrancy) {
            // lerp(c^(1/gamma), l, 1) = l; an infinite channel gives NaN (0) as inf + (inf - inf) does
            lr += col.x - col.x;
            lgc += col.y - col.y;
            lb += col.z - col.z;
        } else
#endif
        {
            lr = lerpf(powf(col.x, inv_gamma_f), lr, vibrancy);
            lgc = lerpf(powf(col.y, inv_gamma_f), lgc, vibrancy);
            lb = lerpf(powf(col.z, inv_gamma_f), lb, vibrancy);
        }
        float a = 0.0f;
        if (C == 4) a = __saturatef(logf(input_density) * log_div / 96.0f);
        pixel_out<C, HALF>::store(out, i, __saturatef(lr), __saturatef(lgc), __saturatef(lb), a);
    }
    if (hist) counts.flush(my_max, hist, max_density);
}

#ifdef RFK_TONEMAP_FAST
inline pow_table make_pow_table(float gamma) {
    static const pow_table base = [] {
        pow_table p{};
        for (int j = 0; j < 32; j++) {
            const double v = std::exp2(j / 32.0);
            p.t[j].x = (float)v;
            p.t[j].y = (float)(v - (double)p.t[j].x);
        }
        return p;
    }();
    pow_table p = base;
    const double q = 1.0 / (double)gamma - 1.0;
    p.q.x = (float)q;
    p.q.y = (float)(q - (double)p.q.x);
    return p;
}
#endif

template <bool HALF, int C>
void launch(unsigned blocks, unsigned sms, cudaStream_t s, const float4* bins, void* out, unsigned size, float gamma, float scale_constant,
            float brightness, float vibrancy, float highlight_power, unsigned long long* hist,
            unsigned long long* max_density, const unsigned long long* q_hits, double q_per_hit) {
    // one wave of persistent blocks at most
    if (blocks > sms * kBlocksPerSm) blocks = sms * kBlocksPerSm;
    tonemap_kernel<C, HALF><<<blocks, 256, 0, s>>>(bins, out, size, gamma, scale_constant, brightness, vibrancy,
                                                    highlight_power, hist, max_density, q_hits, q_per_hit
#ifdef RFK_TONEMAP_FAST
                                                    , make_pow_table(gamma)
#endif
    );
}

}  // namespace rfk_tm
