// Memory-bound layers of the denoiser around the tensor-core convolutions.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "unet_kernels.h"

namespace {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ float bf(const bf16 v) { return __bfloat162float(v); }

// Denoiser input of one histogram: 32 bf16 channels per pixel,
//   0: log1p(density) / 8            1-3: mean colour (rgb / density)
//   4: alpha, sat(ln(density) * 4 / ln 2 / 96) as the tonemapper's
//   5: ln(spp) / 8                   6-8: the tonemapped image of the histogram
//   9-31: 0
__global__ void features_kernel(const float4* __restrict__ bins, const float4* __restrict__ base, size_t npx, float spp,
                                bf16* __restrict__ out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npx) return;
    const float4 b = bins[i];
    const float4 t = base[i];
    float f[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const float d = b.w;
    f[0] = log1pf(fmaxf(d, 0.0f)) * 0.125f;
    if (d > 0.0f) {
        f[1] = b.x / d;
        f[2] = b.y / d;
        f[3] = b.z / d;
    }
    f[4] = d >= 1.0f ? fminf(fmaxf(logf(d) * (4.0f / 0.69314718f) / 96.0f, 0.0f), 1.0f) : 0.0f;
    f[5] = logf(fmaxf(spp, 1.0f)) * 0.125f;
    f[6] = t.x;
    f[7] = t.y;
    f[8] = t.z;
    __nv_bfloat162 h[16];
#pragma unroll
    for (int j = 0; j < 5; j++) h[j] = __floats2bfloat162_rn(f[2 * j], f[2 * j + 1]);
#pragma unroll
    for (int j = 5; j < 16; j++) h[j] = __floats2bfloat162_rn(0.0f, 0.0f);
    uint4* o = reinterpret_cast<uint4*>(out + i * 32);
#pragma unroll
    for (int q = 0; q < 4; q++) o[q] = reinterpret_cast<uint4*>(h)[q];
}

// The layers below move 8 channels (16 bytes) per thread; channel counts,
// strides and offsets are multiples of 8 (32 in this network).
__device__ __forceinline__ void ld8(const bf16* p, float (&v)[8]) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float2 f = __bfloat1622float2(h[j]);
        v[2 * j] = f.x;
        v[2 * j + 1] = f.y;
    }
}

__device__ __forceinline__ void st8(bf16* p, const float (&v)[8]) {
    __nv_bfloat162 h[4];
#pragma unroll
    for (int j = 0; j < 4; j++) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
    *reinterpret_cast<uint4*>(p) = *reinterpret_cast<uint4*>(h);
}

// 2x2 average pool of a channel slice: out[n][y][x][c] = mean of in[n][2y..2y+1][2x..2x+1][coff + c].
__global__ void avgpool_kernel(const bf16* __restrict__ in, int h, int w, int cstride, int coff, int c,
                               bf16* __restrict__ out, unsigned total) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int c8 = c / 8, ho = h / 2, wo = w / 2;
    const int q = (int)(i % c8);
    unsigned r = i / c8;
    const int x = (int)(r % wo);
    r /= wo;
    const int y = (int)(r % ho);
    const unsigned n = r / ho;
    const size_t b = (((size_t)n * h + 2 * y) * w + 2 * x) * cstride + coff + q * 8;
    float a[8], v[8];
    ld8(in + b, a);
    ld8(in + b + cstride, v);
#pragma unroll
    for (int j = 0; j < 8; j++) a[j] += v[j];
    ld8(in + b + (size_t)w * cstride, v);
#pragma unroll
    for (int j = 0; j < 8; j++) a[j] += v[j];
    ld8(in + b + (size_t)w * cstride + cstride, v);
#pragma unroll
    for (int j = 0; j < 8; j++) a[j] = 0.25f * (a[j] + v[j]);
    st8(out + (size_t)i * 8, a);
}

// Gradient through a nearest 2x upsample (sum of the 2x2 block of a channel
// slice of g), times the ReLU derivative of the activation, read where it was
// upsampled to (the same slice of cat):
// out[n][y][x][c] = (cat[n][2y][2x][coff + c] > 0) * sum g[n][2y..][2x..][coff + c].
__global__ void up_backward_kernel(const bf16* __restrict__ g, int gcstride, int gcoff, const bf16* __restrict__ cat,
                                   int h, int w, int c, bf16* __restrict__ out, unsigned total) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int c8 = c / 8;
    const int q = (int)(i % c8);
    unsigned r = i / c8;
    const int x = (int)(r % w);
    r /= w;
    const int y = (int)(r % h);
    const unsigned n = r / h;
    const int W = 2 * w;
    const size_t b = (((size_t)n * 2 * h + 2 * y) * W + 2 * x) * gcstride + gcoff + q * 8;
    float a[8], v[8], m[8];
    ld8(g + b, a);
    ld8(g + b + gcstride, v);
#pragma unroll
    for (int j = 0; j < 8; j++) a[j] += v[j];
    ld8(g + b + (size_t)W * gcstride, v);
#pragma unroll
    for (int j = 0; j < 8; j++) a[j] += v[j];
    ld8(g + b + (size_t)W * gcstride + gcstride, v);
    ld8(cat + b, m);
#pragma unroll
    for (int j = 0; j < 8; j++) a[j] = m[j] > 0.0f ? a[j] + v[j] : 0.0f;
    st8(out + (size_t)i * 8, a);
}

// Gradient of a skip activation s (a channel slice of a concatenation) that
// feeds both the concatenation and a 2x2 average pool, times its ReLU
// derivative: out = (s > 0) * (gcat[slice] + gpool[y / 2][x / 2] / 4).
__global__ void skip_backward_kernel(const bf16* __restrict__ gcat, int cstride, int coff, const bf16* __restrict__ gpool,
                                     const bf16* __restrict__ cat, int h, int w, int c, bf16* __restrict__ out,
                                     unsigned total) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int c8 = c / 8;
    const int q = (int)(i % c8);
    unsigned r = i / c8;
    const int x = (int)(r % w);
    r /= w;
    const int y = (int)(r % h);
    const unsigned n = r / h;
    const size_t px = ((size_t)n * h + y) * w + x;
    float sv[8], gc[8], gp[8];
    ld8(cat + px * cstride + coff + q * 8, sv);
    ld8(gcat + px * cstride + coff + q * 8, gc);
    ld8(gpool + (((size_t)n * (h / 2) + y / 2) * (w / 2) + x / 2) * c + q * 8, gp);
#pragma unroll
    for (int j = 0; j < 8; j++) gc[j] = sv[j] > 0.0f ? gc[j] + 0.25f * gp[j] : 0.0f;
    st8(out + (size_t)i * 8, gc);
}

// Mean squared error of the prediction base + out (the network predicts a
// correction of the tonemapped low-spp image) against target, all f32, 4 per
// pixel, and its gradient as bf16 (channels 3..31 zero). A warp takes 32 pixels
// at a time, so that its stores are 512 contiguous bytes; a block adds its
// squares once. 16 images of 512 x 512: 72 us; with an atomic per warp, 64-byte
// strides between the lanes' stores and 32 f32 channels in `out` 321.
__global__ void __launch_bounds__(256) mse_kernel(const float4* __restrict__ out, const float4* __restrict__ base,
                                                  const float4* __restrict__ target, size_t npx, float inv_n,
                                                  uint4* __restrict__ grad, double* __restrict__ loss) {
    const unsigned lane = threadIdx.x & 31u;
    double sum = 0.0;
    for (size_t p0 = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / 32 * 32; p0 < npx; p0 += (size_t)gridDim.x * blockDim.x) {
        const size_t i = p0 + lane;
        uint2 g = make_uint2(0u, 0u);
        if (i < npx) {
            const float4 t = target[i], b = base[i], o = out[i];
            const float d0 = b.x + o.x - t.x, d1 = b.y + o.y - t.y, d2 = b.z + o.z - t.z;
            sum += (double)(d0 * d0 + d1 * d1 + d2 * d2);
            const __nv_bfloat162 h0 = __floats2bfloat162_rn(2.0f * d0 * inv_n, 2.0f * d1 * inv_n);
            const __nv_bfloat162 h1 = __floats2bfloat162_rn(2.0f * d2 * inv_n, 0.0f);
            g = make_uint2(*reinterpret_cast<const unsigned*>(&h0), *reinterpret_cast<const unsigned*>(&h1));
        }
#pragma unroll
        for (unsigned k = 0; k < 4; k++) {
            // 16-byte piece lane % 4 of pixel 8 k + lane / 4
            const unsigned px = 8 * k + lane / 4;
            const unsigned x = __shfl_sync(0xffffffffu, g.x, px), y = __shfl_sync(0xffffffffu, g.y, px);
            if (p0 + px < npx) grad[(p0 + px) * 4 + lane % 4] = lane % 4 ? make_uint4(0u, 0u, 0u, 0u) : make_uint4(x, y, 0u, 0u);
        }
    }
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    __shared__ double part[8];
    if (lane == 0) part[threadIdx.x / 32] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 8; k++) sum += part[k];
        atomicAdd(loss, sum);
    }
}

// Adam (Kingma & Ba 2015) on the f32 master weights [cout][9][cin] and biases of
// all layers in one launch (a launch for the weights and one for the bias of each of
// 15 layers and 30 clears: 180 us of a step, now 28); writes the bf16 copies used by the forward
// ([cout][9][cin]) and input-gradient ([cin][8 - t][cout]) convolutions. Rows /
// columns outside (live_out, live_in) stay zero (padded channels of the first and
// last layer).
struct adam_args {
    rfk_unet_layer l[RFK_UNET_MAX_LAYERS];
    unsigned end[RFK_UNET_MAX_LAYERS];  // blocks up to and with this layer's
    int n;
    float lr, b1, b2, eps, c1, c2;
};

__device__ __forceinline__ float adam_update(const adam_args& p, float x, float& m, float& v, float g) {
    const float mi = p.b1 * m + (1.0f - p.b1) * g;
    const float vi = p.b2 * v + (1.0f - p.b2) * g * g;
    m = mi;
    v = vi;
    return x - p.lr * (mi / p.c1) / (sqrtf(vi / p.c2) + p.eps);
}

__global__ void __launch_bounds__(256) adam_kernel(const __grid_constant__ adam_args p) {
    int k = 0;
    while (blockIdx.x >= p.end[k]) k++;
    const rfk_unet_layer& y = p.l[k];
    const int i = (int)((blockIdx.x - (k ? p.end[k - 1] : 0u)) * blockDim.x + threadIdx.x);
    const int n = y.cout * 9 * y.cin;
    if (i < n) {
        const int ci = i % y.cin, t = (i / y.cin) % 9, co = i / (9 * y.cin);
        float wi = y.w[i];
        if (co < y.live_out && ci < y.live_in) y.w[i] = wi = adam_update(p, wi, y.m[i], y.v[i], y.g[i]);
        else wi = 0.0f;
        const bf16 h = __float2bfloat16(wi);
        static_cast<bf16*>(y.wf)[i] = h;
        static_cast<bf16*>(y.wb)[((size_t)ci * 9 + (8 - t)) * y.cout + co] = h;
    } else if (i - n < y.cout) {
        const int c = i - n;
        y.b[c] = c < y.live_out ? adam_update(p, y.b[c], y.bm[c], y.bv[c], (float)y.bg[c]) : 0.0f;
    }
}

// Prediction (base + network output) to an image in the tonemapper's formats,
// clamped to [0, 1]; alpha from the histogram as the tonemapper's.
template <int CH, bool HALF>
__global__ void to_image_kernel(const float4* __restrict__ net, const float4* __restrict__ base,
                                const float4* __restrict__ bins, size_t npx, void* out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npx) return;
    const float4 o = net[i], b = base[i];
    float v[4] = {fminf(fmaxf(b.x + o.x, 0.0f), 1.0f), fminf(fmaxf(b.y + o.y, 0.0f), 1.0f),
                  fminf(fmaxf(b.z + o.z, 0.0f), 1.0f), 0.0f};
    if (CH == 4) {
        const float d = bins[i].w;
        v[3] = d > 0.0f ? fminf(fmaxf(logf(d) * (4.0f / 0.69314718f) / 96.0f, 0.0f), 1.0f) : 0.0f;
    }
    if (HALF) {
        __half* h = static_cast<__half*>(out) + i * CH;
        for (int j = 0; j < CH; j++) h[j] = __float2half_rn(v[j]);
    } else {
        float* f = static_cast<float*>(out) + i * CH;
        for (int j = 0; j < CH; j++) f[j] = v[j];
    }
}

inline unsigned blocks_for(size_t n, unsigned t = 256) { return (unsigned)((n + t - 1) / t); }

}  // namespace

extern "C" cudaError_t rfk_unet_features(const float4* bins, const float4* base, size_t npx, float spp, void* out,
                                         cudaStream_t s) {
    if (npx == 0) return cudaSuccess;
    features_kernel<<<blocks_for(npx), 256, 0, s>>>(bins, base, npx, spp, static_cast<bf16*>(out));
    return cudaGetLastError();
}

extern "C" cudaError_t rfk_unet_avgpool(const void* in, int n_img, int h, int w, int cstride, int coff, int c, void* out,
                                        cudaStream_t s) {
    const size_t total = (size_t)n_img * (h / 2) * (w / 2) * (c / 8);
    if (h % 2 || w % 2 || total == 0 || c % 8 || cstride % 8 || coff % 8 || total > 0xFFFFFFFFull) return cudaErrorInvalidValue;
    avgpool_kernel<<<blocks_for(total), 256, 0, s>>>(static_cast<const bf16*>(in), h, w, cstride, coff, c,
                                                      static_cast<bf16*>(out), (unsigned)total);
    return cudaGetLastError();
}

extern "C" cudaError_t rfk_unet_up_backward(const void* g, int gcstride, int gcoff, const void* cat, int n_img, int h, int w,
                                            int c, void* out, cudaStream_t s) {
    const size_t total = (size_t)n_img * h * w * (c / 8);
    if (total == 0 || c % 8 || gcstride % 8 || gcoff % 8 || total > 0xFFFFFFFFull) return cudaErrorInvalidValue;
    up_backward_kernel<<<blocks_for(total), 256, 0, s>>>(static_cast<const bf16*>(g), gcstride, gcoff,
                                                          static_cast<const bf16*>(cat), h, w, c, static_cast<bf16*>(out),
                                                          (unsigned)total);
    return cudaGetLastError();
}

extern "C" cudaError_t rfk_unet_skip_backward(const void* gcat, int cstride, int coff, const void* gpool, const void* cat,
                                              int n_img, int h, int w, int c, void* out, cudaStream_t s) {
    const size_t total = (size_t)n_img * h * w * (c / 8);
    if (total == 0 || h % 2 || w % 2 || c % 8 || cstride % 8 || coff % 8 || total > 0xFFFFFFFFull)
        return cudaErrorInvalidValue;
    skip_backward_kernel<<<blocks_for(total), 256, 0, s>>>(static_cast<const bf16*>(gcat), cstride, coff,
                                                            static_cast<const bf16*>(gpool), static_cast<const bf16*>(cat),
                                                            h, w, c, static_cast<bf16*>(out), (unsigned)total);
    return cudaGetLastError();
}

extern "C" cudaError_t rfk_unet_mse(const float4* out, const float4* base, const float4* target, size_t npx, void* grad,
                                    double* loss, cudaStream_t s) {
    if (npx == 0) return cudaSuccess;
    const unsigned blocks = npx / 256 < 152 * 8 ? blocks_for(npx) : 152 * 8;
    mse_kernel<<<blocks, 256, 0, s>>>(out, base, target, npx, 1.0f / (3.0f * (float)npx), static_cast<uint4*>(grad), loss);
    return cudaGetLastError();
}

extern "C" cudaError_t rfk_unet_adam(const rfk_unet_layer* layers, int n, float lr, float b1, float b2, float eps, int step,
                                     cudaStream_t s) {
    if (n <= 0 || n > RFK_UNET_MAX_LAYERS) return cudaErrorInvalidValue;
    adam_args p{};
    p.n = n;
    p.lr = lr;
    p.b1 = b1;
    p.b2 = b2;
    p.eps = eps;
    p.c1 = 1.0f - powf(b1, (float)step);
    p.c2 = 1.0f - powf(b2, (float)step);
    unsigned blocks = 0;
    for (int k = 0; k < n; k++) {
        p.l[k] = layers[k];
        p.end[k] = blocks += blocks_for((size_t)layers[k].cout * (9 * layers[k].cin + 1));
    }
    adam_kernel<<<blocks, 256, 0, s>>>(p);
    return cudaGetLastError();
}

extern "C" cudaError_t rfk_unet_to_image(const float4* net, const float4* base, const float4* bins, size_t npx, void* out,
                                         int format, cudaStream_t s) {
    if (npx == 0) return cudaSuccess;
    switch (format) {
    case 0: to_image_kernel<3, true><<<blocks_for(npx), 256, 0, s>>>(net, base, bins, npx, out); break;
    case 1: to_image_kernel<4, true><<<blocks_for(npx), 256, 0, s>>>(net, base, bins, npx, out); break;
    case 2: to_image_kernel<3, false><<<blocks_for(npx), 256, 0, s>>>(net, base, bins, npx, out); break;
    case 3: to_image_kernel<4, false><<<blocks_for(npx), 256, 0, s>>>(net, base, bins, npx, out); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}
