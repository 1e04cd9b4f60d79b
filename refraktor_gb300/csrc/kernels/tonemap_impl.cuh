// Tonemap kernel body shared by two translation units: image.cu compiles it
// with full-precision math (PRECISE) and tonemap_fast.cu with -use_fast_math,
// the way the reference builds assets/kernels/tonemap.cu
// (src/librefrakt/src/image/tonemapper.cpp:10-22), so that the fast variant
// matches the reference kernel.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "image_kernels.h"
#include "pow_pair.h"

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
// and gamma >= 1 (the usual genome) the precise build's short form leaves out the
// three c^(1/gamma) whose weight is 0, and the next pixel's load is in flight while
// this one is computed. 1920 x 1080 half4, every pixel lit: 18.5 us a call, 32.9 with
// all four powf. The other form is bound by these: no load ahead and up to 8 blocks
// for an SM's 6 (one kernel for both, as the short form: 34.9 us, 640 x 360 8.2 and 6.3).
struct tonemap_args {
    void* out;
    float gamma, scale_constant, brightness, vibrancy, highlight_power;
};

// SHORT, fast build: the factor w^(1/gamma) / w by pow_pair; false where a channel's
// rounding is left open, and nothing is stored. SHORT, precise build: vibrancy is 1
// and gamma 1 or more.
template <int C, bool HALF, bool SHORT>
__device__ __forceinline__ bool tonemap_pixel(const tonemap_args& p, size_t i, float4 col, const float2* table, float2 q) {
    if (col.w == 0.0f) {
        pixel_out<C, HALF>::store(p.out, i, 0.0f, 0.0f, 0.0f, 0.0f);
        return true;
    }
    const float log_div = 4.0f / logf(2.0f);
    const double inv_gamma = 1.0 / (double)p.gamma;
    const float inv_gamma_f = (float)inv_gamma;
    const float input_density = col.w;
#ifdef RFK_TONEMAP_FAST
    float lg = logf(1.0f + col.w * p.scale_constant);
#else
    float lg = log1pf(col.w * p.scale_constant);
#endif
    const float factor = 0.5f * p.brightness * lg * 0.434294481903251827651128918916f / col.w;
    col.x *= factor;
    col.y *= factor;
    col.z *= factor;
    col.w *= factor;
    float lr, lgc, lb;
#ifdef RFK_TONEMAP_FAST
    if (SHORT) {
        float hi, lo;
        if (!pow_pair(col.w, table, q, hi, lo)) return false;
        bool done = scale_pair(col.x, hi, lo, lr);
        done &= scale_pair(col.y, hi, lo, lgc);
        done &= scale_pair(col.z, hi, lo, lb);
        if (!done) return false;
    } else {
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
    if (p.highlight_power >= 0.0f) highlight(lr, lgc, lb, p.highlight_power);
#ifndef RFK_TONEMAP_FAST
    if (SHORT) {
        // lerp(c^(1/gamma), l, 1) = l, and NaN (0) where c^(1/gamma) is infinite or NaN: for an
        // infinite c, and a negative one unless gamma is 1 (a highlight lifts its l above 0)
        const float negative = inv_gamma_f < 1.0f ? nanf("") : 0.0f;
        lr += col.x < 0.0f ? negative : col.x - col.x;
        lgc += col.y < 0.0f ? negative : col.y - col.y;
        lb += col.z < 0.0f ? negative : col.z - col.z;
    } else
#endif
    {
        lr = lerpf(powf(col.x, inv_gamma_f), lr, p.vibrancy);
        lgc = lerpf(powf(col.y, inv_gamma_f), lgc, p.vibrancy);
        lb = lerpf(powf(col.z, inv_gamma_f), lb, p.vibrancy);
    }
    float a = 0.0f;
    if (C == 4) a = __saturatef(logf(input_density) * log_div / 96.0f);
    pixel_out<C, HALF>::store(p.out, i, __saturatef(lr), __saturatef(lgc), __saturatef(lb), a);
    return true;
}

#ifdef RFK_TONEMAP_FAST
// Out of line: the FP64 power's registers stay out of the pixels' loop.
template <int C, bool HALF>
__device__ __noinline__ void tonemap_pixel_fp64(tonemap_args p, size_t i, float4 col) {
    tonemap_pixel<C, HALF, false>(p, i, col, nullptr, make_float2(0.0f, 0.0f));
}
#endif

// SHORT, fast build: pixels that pow_pair leaves open are put aside, 1 in 120, and
// done by whole warps in FP64 at the block's end; where more come than kOpenPixels (one
// colour everywhere, densities past pow_pair's range) the rest are done at once.
// 1366 x 768 float4 with its histogram: 21 us a call, 98 with every power in FP64 (19.5
// with the pair's roundings taken as they come, 3 in 100000 of them an ulp off).
constexpr unsigned kOpenPixels = 1024;
#ifdef RFK_TONEMAP_FAST
constexpr int kBlocksPerSm = 4;
#else
constexpr int kBlocksPerSm = 6;
#endif

template <int C, bool HALF, bool SHORT>
__global__ void __launch_bounds__(256, kBlocksPerSm)
    tonemap_kernel(const float4* __restrict__ bins, unsigned size, tonemap_args p, unsigned long long* __restrict__ hist,
                   unsigned long long* __restrict__ max_density, const unsigned long long* __restrict__ q_hits, double q_per_hit
#ifdef RFK_TONEMAP_FAST
                   , const __grid_constant__ pow_table pt
#endif
    ) {
    __shared__ density_counts counts;
    if (hist) counts.clear();
    float2 *table = nullptr, q = {0.0f, 0.0f};
#ifdef RFK_TONEMAP_FAST
    __shared__ float2 table_sm[32];
    __shared__ unsigned open[SHORT ? kOpenPixels : 1], nopen;
    if (SHORT) {
        if (threadIdx.x < 32) table_sm[threadIdx.x] = pt.t[threadIdx.x];
        if (threadIdx.x == 0) nopen = 0;
        __syncthreads();
        table = table_sm;
        q = pt.q;
    }
#endif
    if (q_hits) {
        // quality from a device counter (batched renders): the host constant
        // of the single-image path, computed here in single precision
        const float quality = (float)((double)*q_hits * q_per_hit);
        p.scale_constant = powf(10.0f, -log10f(quality) - 0.5f);
    }
    const float log_div = 4.0f / logf(2.0f);
    float my_max = 0.0f;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    float4 next = SHORT && i < size ? bins[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (; i < size; i += stride) {
        const float4 col = SHORT ? next : bins[i];
        if (SHORT && i + stride < size) next = bins[i + stride];
        if (hist) {
            atomicAdd(&counts.bins[density_counts::bin(col.w, log_div)], 1u);
            if (col.w >= 1.0f) my_max = fmaxf(my_max, col.w);
        }
        const bool done = tonemap_pixel<C, HALF, SHORT>(p, i, col, table, q);
        (void)done;
#ifdef RFK_TONEMAP_FAST
        if (SHORT && !done) {
            const unsigned at = atomicAdd(&nopen, 1u);
            if (at < kOpenPixels) open[at] = (unsigned)i;
            else tonemap_pixel_fp64<C, HALF>(p, i, col);
        }
#endif
    }
#ifdef RFK_TONEMAP_FAST
    if (SHORT) {
        __syncthreads();
        const unsigned n = min(nopen, kOpenPixels);
        for (unsigned k = threadIdx.x; k < n; k += blockDim.x) tonemap_pixel_fp64<C, HALF>(p, open[k], bins[open[k]]);
    }
#endif
    if (hist) counts.flush(my_max, hist, max_density);
}

template <bool HALF, int C, bool SHORT>
void launch_form(unsigned blocks, unsigned sms, cudaStream_t s, const float4* bins, unsigned size, const tonemap_args& p,
                 unsigned long long* hist, unsigned long long* max_density, const unsigned long long* q_hits, double q_per_hit) {
    // persistent blocks: one wave at most in the short form
    const unsigned cap = sms * (SHORT ? kBlocksPerSm : 8);
    if (blocks > cap) blocks = cap;
    tonemap_kernel<C, HALF, SHORT><<<blocks, 256, 0, s>>>(bins, size, p, hist, max_density, q_hits, q_per_hit
#ifdef RFK_TONEMAP_FAST
                                                          , SHORT ? make_pow_table(p.gamma) : pow_table{}
#endif
    );
}

template <bool HALF, int C>
void launch(unsigned blocks, unsigned sms, cudaStream_t s, const float4* bins, void* out, unsigned size, float gamma, float scale_constant,
            float brightness, float vibrancy, float highlight_power, unsigned long long* hist,
            unsigned long long* max_density, const unsigned long long* q_hits, double q_per_hit) {
    const tonemap_args p{out, gamma, scale_constant, brightness, vibrancy, highlight_power};
#ifdef RFK_TONEMAP_FP64
    const bool is_short = false;
#elif defined(RFK_TONEMAP_FAST)
    const bool is_short = gamma >= kPowPairGamma;
#else
    const bool is_short = vibrancy == 1.0f && gamma >= 1.0f;
#endif
    if (is_short) {
        launch_form<HALF, C, true>(blocks, sms, s, bins, size, p, hist, max_density, q_hits, q_per_hit);
    } else {
        launch_form<HALF, C, false>(blocks, sms, s, bins, size, p, hist, max_density, q_hits, q_per_hit);
    }
}

}  // namespace rfk_tm
