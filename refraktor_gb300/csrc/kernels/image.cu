// Flame-independent kernels of the render path, compiled by nvcc for sm_103a:
// Catmull-Rom segment coefficients, log-density tonemap (with the density
// histogram of the reference fused into the same pass), the stand-alone
// density histogram, the density-estimation blur, and two roofline probes.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>

#include "image_kernels.h"

namespace {

// ------------------------------------------------------------ Catmull-Rom --
// Centripetal Catmull-Rom (alpha = 0.5, tension 0) segment p1 -> p2 with knot
// distance sqrt(hypot(dp, 1)), as assets/kernels/catmull.cu:11-28, evaluated
// in FP32 from the FP64 packed samples and stored in Hermite form
// (p1, p2, m1, m2). One thread per (segment, real).
__global__ void __launch_bounds__(256) catmull_kernel(const double* __restrict__ samples, unsigned sample_size,
                                                      unsigned nseg, float4* __restrict__ coeff) {
    const unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (unsigned long long)sample_size * nseg) return;
    const unsigned seg = (unsigned)(i / sample_size), r = (unsigned)(i % sample_size);
    const size_t base = (size_t)seg * sample_size + r;
    const float p0 = (float)samples[base], p1 = (float)samples[base + sample_size];
    const float p2 = (float)samples[base + 2 * (size_t)sample_size], p3 = (float)samples[base + 3 * (size_t)sample_size];
    const float t01 = sqrtf(hypotf(p1 - p0, 1.0f));
    const float t12 = sqrtf(hypotf(p2 - p1, 1.0f));
    const float t23 = sqrtf(hypotf(p3 - p2, 1.0f));
    const float m1 = p2 - p1 + t12 * ((p1 - p0) / t01 - (p2 - p0) / (t01 + t12));
    const float m2 = p2 - p1 + t12 * ((p3 - p2) / t23 - (p3 - p1) / (t12 + t23));
    // Hermite form: a = 2(p1-p2)+m1+m2, b = -3(p1-p2)-2m1-m2, c = m1, d = p1
    // of the reference describe the same cubic
    coeff[i] = make_float4(p1, p2, m1, m2);
}

// ----------------------------------------------------------------- tonemap --
// (kernel text in tonemap_impl.cuh; the fast variant lives in tonemap_fast.cu)
#include "tonemap_impl.cuh"

// ------------------------------------------------------- density histogram --
__global__ void __launch_bounds__(256) density_histogram_kernel(const float4* __restrict__ bins, unsigned size,
                                                                unsigned long long* __restrict__ hist,
                                                                unsigned long long* __restrict__ max_density) {
    __shared__ rfk_tm::density_counts counts;
    counts.clear();
    const float log_div = 4.0f / logf(2.0f);
    float my_max = 0.0f;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
#pragma unroll 4
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < size; i += stride) {
        const float v = bins[i].w;
        atomicAdd(&counts.bins[rfk_tm::density_counts::bin(v, log_div)], 1u);
        if (v >= 1.0f) my_max = fmaxf(my_max, v);
    }
    counts.flush(my_max, hist, max_density);
}

// -------------------------------------------------- density-estimation blur --
// Each source pixel q with density d > 0 spreads its RGBA over a disc of radius
//   r(q) = clamp(max_radius * d^(-curve), min_radius, max_radius)
// quantised to 1/RFK_DE_STEPS px; the weight of integer offset o is
//   k(o) = max(0, 1 - |o|^2 / (r + 1)^2) / Z(r),  Z(r) = sum over |ox|,|oy| <= ceil(r) of the same,
// so a pixel of radius 0 keeps its value and every source conserves its total
// (inside the image).
//
// A block owns a strip of 32 output columns (lane = column) and walks down its
// source rows, the strip's rows and a halo of 9, eight rows a step, one per
// warp. What bounds the kernel is the FP32 work per (source, output) pair - an
// fma for k, a max, four fmas - so a step does it once for both output rows at
// distance d = 0 .. 9 of a source row:
//   H[d] = sum over the row's sources of v max(0, 1 - (dx^2 + d^2) a) / Z
// goes through shared memory to the rows above and below, whose sums wait in
// registers (the warp keeps every eighth output row) until the walk has passed
// them. H takes few pairs that are zero:
//   - sources that reach at most 2 px (the bulk of a converged image) are
//     gathered, five taps per source row, each lane its own sources;
//   - wider sources are taken one by one from the row's bit mask, all lanes on
//     the same source (its values broadcast from shared memory), distances
//     beyond its reach skipped three at a time. A real 1080p frame has 20-35%
//     such sources; a pixel is reached by 20-100 of the 361 in its window;
//   - a row with more of them than taps is gathered over its full reach.
// Measured (GB300): a 1024-spp 1920 x 1080 frame 162 us, a 1280 x 720 animation
// frame 75-79 us, a faint 256 x 256 image 21 us; one thread per pixel looping
// over a shared tile up to the tile's widest reach took 632, 208-330 and 90 us.
// 8 warps x 3 blocks per SM (80 registers) issue 75% of the slots.
#define DE_HALO 9  // RFK_DE_MAX_RADIUS_CAP
#define DE_WARPS 8  // source rows a step
#define DE_TILE_X 32
#define DE_SW (DE_TILE_X + 2 * DE_HALO)
#define DE_SMALL 2  // reach of the sources that are gathered

// Per radius level: 1 / (r + 1)^2, rounded up where that keeps the offset
// ceil(r) + 1 at weight 0, 1 / Z(r), and ceil(r).
struct de_table {
    float a[RFK_DE_LEVELS], inv_z[RFK_DE_LEVELS];
    int reach[RFK_DE_LEVELS];
};

// Radius level (r * RFK_DE_STEPS) of a source pixel of density d > 0.
__device__ __forceinline__ int de_level(float d, float max_radius, float min_radius, float curve) {
    float r = max_radius * powf(d, -curve);
    r = fminf(fmaxf(r, min_radius), max_radius);
    return (int)(unsigned char)lrintf(r * RFK_DE_STEPS);
}

// One source row of a warp's strip: columns -9 .. 40 of it.
struct de_row {
    float4 v[DE_SW];  // RGBA / Z, 0 where there is no source
    float a[DE_SW];   // 1 / (r + 1)^2
    unsigned char reach[DE_SW + 2];
};

// p += q k for two channels in one instruction (the kernel issues 75% of its
// slots: 5 instead of 6 instructions a pair took a 1080p frame from 174 to 162 us).
__device__ __forceinline__ void fma_pair(float& px, float& py, float qx, float qy, float k) {
    unsigned long long p, q, kk;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(px), "f"(py));
    asm("mov.b64 %0, {%1, %2};" : "=l"(q) : "f"(qx), "f"(qy));
    asm("mov.b64 %0, {%1, %1};" : "=l"(kk) : "f"(k));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(p) : "l"(q), "l"(kk));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(px), "=f"(py) : "l"(p));
}

// H[d] += v k(dx, d) for d = D0 .. D1; t = 1 - dx^2 a. A non-finite source is
// added where k > 0 only, so that it stays inside its own support.
template <bool FINITE, int D0, int D1>
__device__ __forceinline__ void de_add(float4 (&H)[DE_HALO + 1], const float4& v, float a, float t) {
#pragma unroll
    for (int d = D0; d <= D1; d++) {
        float k = fmaf(-(float)(d * d), a, t);
        if (FINITE) k = fmaxf(k, 0.0f);
        if (FINITE || k > 0.0f) {
            fma_pair(H[d].x, H[d].y, v.x, v.y, k);
            fma_pair(H[d].z, H[d].w, v.z, v.w, k);
        }
    }
}

template <bool FINITE>
__device__ __forceinline__ void de_add_reach(float4 (&H)[DE_HALO + 1], const float4& v, float a, float t, int reach) {
    de_add<FINITE, 0, 3>(H, v, a, t);
    if (reach > 3) de_add<FINITE, 4, 6>(H, v, a, t);
    if (reach > 6) de_add<FINITE, 7, DE_HALO>(H, v, a, t);
}

// H of the row's wide sources (mask: their columns, reach: the widest).
template <bool FINITE>
__device__ __forceinline__ void de_wide(const de_row& row, int lane, unsigned long long mask, int reach, float4 (&H)[DE_HALO + 1]) {
    const float wide_a = 1.0f / ((DE_SMALL + 1) * (DE_SMALL + 1));  // a of a source is below it if it is wide
    if (__popcll(mask) > 2 * reach) {
#pragma unroll 1
        for (int dx = -reach; dx <= reach; dx++) {
            const int c = lane + DE_HALO + dx;
            const float a = row.a[c];
            const float4 v = row.v[c];
            de_add_reach<FINITE>(H, v, a, a < wide_a ? fmaf((float)(-dx * dx), a, 1.0f) : 0.0f, reach);
        }
        return;
    }
#pragma unroll 1
    while (mask) {
        const int c = __ffsll((long long)mask) - 1;
        mask &= mask - 1ull;
        const int rc = row.reach[c];
        if (rc < max(DE_HALO - c, c - (DE_HALO + DE_TILE_X - 1))) continue;  // short of the strip
        const float a = row.a[c];
        const float4 v = row.v[c];
        const float dx = (float)(lane + DE_HALO - c);
        de_add_reach<FINITE>(H, v, a, fmaf(-dx * dx, a, 1.0f), rc);
    }
}

// H[0 .. 2] of the sources that reach at most DE_SMALL.
template <bool FINITE>
__device__ __forceinline__ void de_small(const de_row& row, int lane, float4 (&H)[DE_HALO + 1]) {
    const float wide_a = 1.0f / ((DE_SMALL + 1) * (DE_SMALL + 1));
#pragma unroll
    for (int dx = -DE_SMALL; dx <= DE_SMALL; dx++) {
        const int c = lane + DE_HALO + dx;
        const float a = row.a[c];
        const float4 v = row.v[c];
        de_add<FINITE, 0, DE_SMALL>(H, v, a, a < wide_a ? 0.0f : fmaf((float)(-dx * dx), a, 1.0f));
    }
}

__global__ void __launch_bounds__(32 * DE_WARPS, 3) de_blur_kernel(const float4* __restrict__ in, float4* __restrict__ out,
                                                                   unsigned w, unsigned h, float max_radius, float min_radius,
                                                                   float curve, int steps, const __grid_constant__ de_table tab) {
    __shared__ union {
        de_row row;                          // the warp's source row, then
        float4 H[DE_HALO + 1][DE_TILE_X];    // its H
    } sm[DE_WARPS];
    __shared__ int reach_sm[DE_WARPS];       // H[0 .. reach] is set; -1: the row has no source
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    de_row& row = sm[warp].row;
    const int rows = steps * DE_WARPS - 2 * DE_HALO;
    const int y0 = (int)blockIdx.y * rows, y1 = min((int)h, y0 + rows);
    const int x0 = blockIdx.x * DE_TILE_X - DE_HALO;
    const int gx = x0 + DE_HALO + lane;

    // the warp's source row s: columns lane and lane + 32 (the last 18) of the strip's window
    const bool in0 = x0 + lane >= 0 && x0 + lane < (int)w;
    const bool in1 = lane < DE_SW - 32 && x0 + lane + 32 < (int)w;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 n0 = zero, n1 = zero;
    auto fetch = [&](int s) {
        n0 = n1 = zero;
        if (s < 0 || s >= (int)h) return;
        const float4* src = in + (size_t)s * w + x0 + lane;
        if (in0) n0 = src[0];
        if (in1) n1 = src[32];
    };
    // sums of output rows s0 + own + 8 i, of those the step's rows s0 .. s0 + 7
    // reach; the first is complete after the step
    const int own = warp == DE_WARPS - 1 ? -1 : warp;
    float4 B[4] = {zero, zero, zero, zero};
    fetch(y0 - DE_HALO + warp);
#pragma unroll 1
    for (int step = 0; step < steps; step++) {
        const int s0 = y0 - DE_HALO + step * DE_WARPS;
        unsigned long long wide = 0ull;
        unsigned small = 0u, odd = 0u, widest = 0u;
#pragma unroll
        for (int half = 0; half < 2; half++) {
            float4 v = half ? n1 : n0;
            int reach = 0;
            float a = 1.0f;
            const bool source = v.w > 0.0f;
            if (source) {
                const int l = de_level(v.w, max_radius, min_radius, curve);
                const float z = tab.inv_z[l];
                a = tab.a[l];
                reach = tab.reach[l];
                v = make_float4(v.x * z, v.y * z, v.z * z, v.w * z);
            } else {
                v = zero;
            }
            const int c = lane + 32 * half;
            if (c < DE_SW) {
                row.v[c] = v;
                row.a[c] = a;
                row.reach[c] = (unsigned char)reach;
            }
            wide |= (unsigned long long)__ballot_sync(0xffffffffu, reach > DE_SMALL) << (32 * half);
            small |= __ballot_sync(0xffffffffu, source && reach <= DE_SMALL);
            odd |= __ballot_sync(0xffffffffu, !(isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w)));
            widest = max(widest, __reduce_max_sync(0xffffffffu, (unsigned)reach));
        }
        __syncwarp();
        fetch(s0 + DE_WARPS + warp);
        const int reach = wide ? (int)widest : small ? DE_SMALL : -1;
        if (reach >= 0) {
            float4 H[DE_HALO + 1];
#pragma unroll
            for (int d = 0; d <= DE_HALO; d++) H[d] = zero;
            if (odd) {
                if (small) de_small<false>(row, lane, H);
                if (wide) de_wide<false>(row, lane, wide, reach, H);
            } else {
                if (small) de_small<true>(row, lane, H);
                if (wide) de_wide<true>(row, lane, wide, reach, H);
            }
            __syncwarp();  // H takes the row's place
#pragma unroll
            for (int d = 0; d <= DE_HALO; d++)
                if (d <= reach) sm[warp].H[d][lane] = H[d];
        }
        if (lane == 0) reach_sm[warp] = reach;
        __syncthreads();
#pragma unroll
        for (int s = 0; s < DE_WARPS; s++) {
            const int rs = reach_sm[s];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int d = abs(own + 8 * (i - 1) - s);
                if (d <= rs) {
                    const float4 q = sm[s].H[d][lane];
                    B[i].x += q.x;
                    B[i].y += q.y;
                    B[i].z += q.z;
                    B[i].w += q.w;
                }
            }
        }
        const int y = s0 + own - DE_WARPS;
        if (y >= y0 && y < y1 && gx < (int)w) out[(size_t)y * w + gx] = B[0];
        B[0] = B[1];
        B[1] = B[2];
        B[2] = B[3];
        B[3] = zero;
        __syncthreads();
    }
}

// ------------------------------------------------------------------ probes --
// Throughput of red.global.add.v4.f32 to pseudo-random float4 slots of a
// buffer: the L2-atomic roofline of the histogram update.
__global__ void red_v4_probe_kernel(float4* __restrict__ buf, unsigned long long n, unsigned iters, unsigned seed) {
    unsigned x = (blockIdx.x * blockDim.x + threadIdx.x) * 2654435761u + seed;
    for (unsigned i = 0; i < iters; i++) {
        x ^= x << 13;
        x ^= x >> 17;
        x ^= x << 5;
        const unsigned long long idx = ((unsigned long long)x * n) >> 32;
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(buf + idx), "f"(1.0f), "f"(0.5f), "f"(0.25f),
                     "f"(1.0f)
                     : "memory");
    }
}

// Issue-rate probes of the two arithmetic pipes the chain step leans on:
// pipe 0 = FP32 FMA (8 independent fmaf chains per thread), pipe 1 = the
// special-function unit (sin.approx and rsqrt.approx, 8 independent chains:
// sin(x) stays in [-1, 1] and rsqrt of a positive value converges to 1, so no
// chain reaches inf or NaN). Each thread stores its sum so that nothing is
// dead code.
__global__ void pipe_probe_kernel(float* __restrict__ out, unsigned iters, int pipe) {
    const unsigned gid = blockIdx.x * blockDim.x + threadIdx.x;
    float a[8];
#pragma unroll
    for (int j = 0; j < 8; j++) a[j] = 0.5f + 0.001f * (float)((gid + j) & 255);
    if (pipe == 0) {
        for (unsigned i = 0; i < iters; i++) {
#pragma unroll
            for (int j = 0; j < 8; j++) a[j] = fmaf(a[j], 0.9999f, 0.0001f);
        }
    } else {
        for (unsigned i = 0; i < iters; i++) {
#pragma unroll
            for (int j = 0; j < 4; j++) asm volatile("sin.approx.ftz.f32 %0, %0;" : "+f"(a[j]));
#pragma unroll
            for (int j = 4; j < 8; j++) asm volatile("rsqrt.approx.ftz.f32 %0, %0;" : "+f"(a[j]));
        }
    }
    float sum = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; j++) sum += a[j];
    out[gid] = sum;
}

// ---------------------------------------------------------------- convert --
// convert_to<In, Out> of assets/kernels/convert.cu:70-99: half3 / half4 in,
// uchar3 / uchar4 / float3 / float4 out; a byte is min(v * 255, 255)
// truncated; flip_y writes row h-1-y, swap_channels exchanges R and B; a
// 4-channel output of a 3-channel input gets alpha 1.
// The reference multiplies in double; a half times 255 has at most 19
// significant bits, so the FP32 product is the same number, and the kernel is
// left to memory: a thread takes 4 pixels with 8- or 16-byte loads and 4- or
// 16-byte stores where they are aligned (not to float4 or small float3 images), else
// one pixel. 3840 x 2160 half4 to uchar3: 16.6 us; 230 us with FP64 and one pixel a
// thread.
template <int CIN>
__device__ __forceinline__ void convert_load(const __half* p, int swap, float (&v)[4]) {
#pragma unroll
    for (int c = 0; c < 4; c++) v[c] = c < CIN ? __half2float(p[c]) : 1.0f;
    if (swap) {
        const float t = v[0];
        v[0] = v[2];
        v[2] = t;
    }
}

template <int COUT, bool BYTES>
__device__ __forceinline__ void convert_store(void* out, const float (&v)[4]) {
#pragma unroll
    for (int c = 0; c < COUT; c++) {
        if (BYTES) {
            const float b = fminf(v[c] * 255.0f, 255.0f);  // NaN becomes 255, as fmin in double
            static_cast<unsigned char*>(out)[c] = (unsigned char)(b > 0.0f ? b : 0.0f);
        } else {
            static_cast<float*>(out)[c] = v[c];
        }
    }
}

template <int CIN, int COUT, bool BYTES, bool VEC>
__global__ void __launch_bounds__(256) convert_kernel(const __half* __restrict__ in, void* __restrict__ out, unsigned w,
                                                      unsigned h, int flip_y, int swap) {
    constexpr unsigned OUT = COUT * (BYTES ? 1 : 4);  // bytes of an output pixel
    const unsigned n = w * h;
    float v[4];
    if (!VEC) {
        const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
        if (i >= n) return;
        convert_load<CIN>(in + (size_t)i * CIN, swap, v);  // on its way while the row is worked out
        unsigned o = i;
        if (flip_y) o = (h - i / w - 1) * w + i % w;
        convert_store<COUT, BYTES>(static_cast<unsigned char*>(out) + (size_t)o * OUT, v);
        return;
    }
    constexpr unsigned PX = 4;
    const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * PX;
    if (i >= n) return;
    size_t o = i;  // with flip_y a group of 4 stays within a row (w % 4 == 0)
    if (flip_y) o = (size_t)(h - (unsigned)i / w - 1) * w + (unsigned)i % w;
    unsigned char* dst = static_cast<unsigned char*>(out) + o * OUT;
    if (i + PX <= n) {
        __align__(16) __half p[PX * CIN];
        if (CIN == 4) {
            const uint4* src = reinterpret_cast<const uint4*>(in + i * CIN);
            reinterpret_cast<uint4*>(p)[0] = src[0];
            reinterpret_cast<uint4*>(p)[1] = src[1];
        } else {
            const uint2* src = reinterpret_cast<const uint2*>(in + i * CIN);
#pragma unroll
            for (int q = 0; q < 3; q++) reinterpret_cast<uint2*>(p)[q] = src[q];
        }
        __align__(16) unsigned char r[PX * OUT];
#pragma unroll
        for (unsigned k = 0; k < PX; k++) {
            convert_load<CIN>(p + k * CIN, swap, v);
            convert_store<COUT, BYTES>(r + k * OUT, v);
        }
        if (OUT == 3) {
#pragma unroll
            for (int q = 0; q < 3; q++) reinterpret_cast<unsigned*>(dst)[q] = reinterpret_cast<unsigned*>(r)[q];
        } else {
#pragma unroll
            for (unsigned q = 0; q < PX * OUT / 16; q++) reinterpret_cast<uint4*>(dst)[q] = reinterpret_cast<uint4*>(r)[q];
        }
        return;
    }
    for (unsigned k = 0; k < PX && i + k < n; k++) {
        convert_load<CIN>(in + (i + k) * CIN, swap, v);
        convert_store<COUT, BYTES>(dst + k * OUT, v);
    }
}

template <int CIN, int COUT, bool BYTES>
void launch_convert(const __half* in, void* out, unsigned w, unsigned h, int flip_y, int swap, cudaStream_t s) {
    const size_t n = (size_t)w * h;
    const uintptr_t in_mask = CIN == 4 ? 15 : 7, out_mask = COUT * (BYTES ? 1 : 4) == 3 ? 3 : 15;
    const bool vec = ((uintptr_t)in & in_mask) == 0 && ((uintptr_t)out & out_mask) == 0 && (!flip_y || w % 4 == 0);
    // float4: a pixel fills a 16-byte store by itself (1920 x 1080 half4: 10.6 us, 11.4
    // with 4 pixels a thread); float3: small images lose threads by it (640 x 360 half3:
    // 2.60 us, 2.75 with 4 pixels; 1280 x 720 5.41 and 4.80)
    if constexpr (BYTES || COUT == 3) {
        if (vec && (BYTES || n >= (1u << 19))) {
            convert_kernel<CIN, COUT, BYTES, true><<<(unsigned)((n + 1023) / 1024), 256, 0, s>>>(in, out, w, h, flip_y, swap);
            return;
        }
    }
    convert_kernel<CIN, COUT, BYTES, false><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(in, out, w, h, flip_y, swap);
}

// Counters of a render (rfk_counters: 0, the earliest start the largest value) and
// `n` words in all.
__global__ void clear_counters_kernel(unsigned long long* c, unsigned n) {
    for (unsigned i = threadIdx.x; i < n; i += blockDim.x) c[i] = i == 2 ? ~0ull : 0ull;
}

de_table de_make_table() {
    de_table t;
    for (int l = 0; l < RFK_DE_LEVELS; l++) {
        const float r = (float)l / RFK_DE_STEPS, r1 = (r + 1.0f) * (r + 1.0f);
        const int rc = (l + RFK_DE_STEPS - 1) / RFK_DE_STEPS;
        float a = 1.0f / r1;
        while (std::fma(-(float)((rc + 1) * (rc + 1)), a, 1.0f) > 0.0f) a = std::nextafter(a, 2.0f);
        float z = 0.0f;
        for (int oy = -rc; oy <= rc; oy++)
            for (int ox = -rc; ox <= rc; ox++) z += std::fmax(0.0f, std::fma(-(float)(ox * ox + oy * oy), a, 1.0f));
        t.a[l] = a;
        t.inv_z[l] = 1.0f / z;
        t.reach[l] = rc;
    }
    return t;
}

int sm_count() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 1;
    }
    return n;
}

}  // namespace

extern "C" {

cudaError_t rfk_launch_catmull(const double* samples, unsigned sample_size, unsigned nseg, float4* coeff, cudaStream_t s) {
    const unsigned long long n = (unsigned long long)sample_size * nseg;
    if (n == 0) return cudaSuccess;
    catmull_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(samples, sample_size, nseg, coeff);
    return cudaGetLastError();
}

cudaError_t rfk_launch_tonemap_fast(const float4* bins, unsigned size, void* out, int format, float gamma,
                                    float scale_constant, float brightness, float vibrancy, float highlight_power,
                                    unsigned long long* hist, unsigned long long* max_density,
                                    const unsigned long long* q_hits, double q_per_hit, unsigned blocks, unsigned sms,
                                    cudaStream_t s);

cudaError_t rfk_launch_tonemap(const float4* bins, unsigned size, void* out, int format, int precise, float gamma,
                               float scale_constant, float brightness, float vibrancy, float highlight_power,
                               unsigned long long* hist, unsigned long long* max_density, const unsigned long long* q_hits,
                               double q_per_hit, cudaStream_t s) {
    if (size == 0) return cudaSuccess;
    const unsigned blocks = (unsigned)(((size_t)size + 255) / 256), sms = (unsigned)sm_count();
    if (!precise)
        return rfk_launch_tonemap_fast(bins, size, out, format, gamma, scale_constant, brightness, vibrancy, highlight_power,
                                       hist, max_density, q_hits, q_per_hit, blocks, sms, s);
    switch (format) {
    case 0: rfk_tm::launch<true, 3>(blocks, sms, s, bins, out, size, gamma, scale_constant, brightness, vibrancy, highlight_power, hist, max_density, q_hits, q_per_hit); break;
    case 1: rfk_tm::launch<true, 4>(blocks, sms, s, bins, out, size, gamma, scale_constant, brightness, vibrancy, highlight_power, hist, max_density, q_hits, q_per_hit); break;
    case 2: rfk_tm::launch<false, 3>(blocks, sms, s, bins, out, size, gamma, scale_constant, brightness, vibrancy, highlight_power, hist, max_density, q_hits, q_per_hit); break;
    case 3: rfk_tm::launch<false, 4>(blocks, sms, s, bins, out, size, gamma, scale_constant, brightness, vibrancy, highlight_power, hist, max_density, q_hits, q_per_hit); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t rfk_launch_density_histogram(const float4* bins, unsigned size, unsigned long long* hist,
                                         unsigned long long* max_density, cudaStream_t s) {
    if (size == 0) return cudaSuccess;
    unsigned blocks = (unsigned)(((size_t)size + 255) / 256);
    const unsigned cap = (unsigned)sm_count() * 8;
    if (blocks > cap) blocks = cap;
    density_histogram_kernel<<<blocks, 256, 0, s>>>(bins, size, hist, max_density);
    return cudaGetLastError();
}

cudaError_t rfk_launch_de_blur(const float4* in, float4* out, unsigned w, unsigned h, float max_radius, float min_radius,
                               float curve, cudaStream_t s) {
    if (w == 0 || h == 0) return cudaSuccess;
    static const de_table tab = de_make_table();
    const unsigned strips = (w + DE_TILE_X - 1) / DE_TILE_X;
    // steps per block: more of them share the halo, fewer spread the rows over
    // the SMs. A step of a block takes about as long as its share of the SM, but
    // no less than that of one block alone. (512 x 512: 6 steps 41 us, 16 steps
    // 76 us; 1920 x 1080: 4 steps 268 us, 12 steps 174 us.)
    int steps = 3;
    double best = 1e30;
    for (int n = 3; n <= 24; n++) {
        const unsigned rows = (unsigned)(n * DE_WARPS - 2 * DE_HALO);
        const double per_sm = (double)strips * ((h + rows - 1) / rows) / sm_count();
        const double cost = n * ((per_sm > 1.0 ? per_sm : 1.0) + 1.0);
        if (cost < best) {
            best = cost;
            steps = n;
        }
    }
    const unsigned rows = (unsigned)(steps * DE_WARPS - 2 * DE_HALO);
    const dim3 grid(strips, (h + rows - 1) / rows);
    de_blur_kernel<<<grid, 32 * DE_WARPS, 0, s>>>(in, out, w, h, max_radius, min_radius, curve, steps, tab);
    return cudaGetLastError();
}

cudaError_t rfk_launch_red_v4_probe(float4* buf, unsigned long long n, unsigned iters, unsigned blocks, unsigned threads,
                                    cudaStream_t s) {
    red_v4_probe_kernel<<<blocks, threads, 0, s>>>(buf, n, iters, 12345u);
    return cudaGetLastError();
}

cudaError_t rfk_launch_pipe_probe(float* out, unsigned iters, int pipe, unsigned blocks, unsigned threads,
                                  cudaStream_t s) {
    pipe_probe_kernel<<<blocks, threads, 0, s>>>(out, iters, pipe);
    return cudaGetLastError();
}

cudaError_t rfk_launch_convert(const void* in, int in_channels, void* out, int out_format, unsigned w, unsigned h,
                               int flip_y, int swap, cudaStream_t s) {
    if (w == 0 || h == 0) return cudaSuccess;
    const __half* src = static_cast<const __half*>(in);
    // out_format: 2 float3, 3 float4, 4 uchar3, 5 uchar4
    if (in_channels == 3) {
        switch (out_format) {
        case 2: launch_convert<3, 3, false>(src, out, w, h, flip_y, swap, s); break;
        case 3: launch_convert<3, 4, false>(src, out, w, h, flip_y, swap, s); break;
        case 4: launch_convert<3, 3, true>(src, out, w, h, flip_y, swap, s); break;
        case 5: launch_convert<3, 4, true>(src, out, w, h, flip_y, swap, s); break;
        default: return cudaErrorInvalidValue;
        }
    } else if (in_channels == 4) {
        switch (out_format) {
        case 2: launch_convert<4, 3, false>(src, out, w, h, flip_y, swap, s); break;
        case 3: launch_convert<4, 4, false>(src, out, w, h, flip_y, swap, s); break;
        case 4: launch_convert<4, 3, true>(src, out, w, h, flip_y, swap, s); break;
        case 5: launch_convert<4, 4, true>(src, out, w, h, flip_y, swap, s); break;
        default: return cudaErrorInvalidValue;
        }
    } else {
        return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t rfk_launch_clear_counters(unsigned long long* c, unsigned n, cudaStream_t s) {
    clear_counters_kernel<<<1, 128, 0, s>>>(c, n);
    return cudaGetLastError();
}

}  // extern "C"
