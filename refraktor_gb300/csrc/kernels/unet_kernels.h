// Launchers of the denoiser kernels (unet_tc.cu: tensor-core convolutions,
// unet_ops.cu: the memory-bound layers around them). Activations are bf16
// NHWC tensors addressed as (pointer, channels per pixel = cstride, channel
// offset = coff), so a layer can read or write a channel slice of a wider
// tensor (the U-Net's concatenations are written in place).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#define RFK_UNET_RELU 1    // conv epilogue: ReLU after the bias
#define RFK_UNET_F32OUT 2  // conv epilogue: store f32 instead of bf16
#define RFK_UNET_UP2 4     // conv epilogue: store each output pixel at its 2x2 pixels of a (2h, 2w) output
                           // (nearest upsampling into the next level's concatenation; bf16, no accumulate)
#define RFK_UNET_RGBOUT 16  // conv epilogue: store the first four channels as f32 (cstride 4)

#define RFK_UNET_MAX_LAYERS 24

// A layer's f32 master weights [cout][9][cin] and bias with their Adam moments and
// gradients, and its bf16 copies wf [cout][9][cin] and wb [cin][9][cout].
struct rfk_unet_layer {
    float *w, *m, *v;
    const float* g;
    float *b, *bm, *bv;
    const double* bg;
    void *wf, *wb;
    int cin, cout, live_in, live_out;
};

#ifdef __cplusplus
extern "C" {
#endif

// 3x3 convolution, stride 1, zero padding 1, on tcgen05: out[:, :, :, coff:coff+cout] (=|+=) epilogue(
// conv(in[..., in_coff:in_coff+cin], weights[cout][9][cin]) + bias) with optional ReLU (flags) and
// multiplication by (mask > 0). Channel counts and offsets are multiples of 32; tensors 64-byte
// aligned. *err is set to 1 if a pipeline wait of the kernel ran out of time.
cudaError_t rfk_unet_conv3x3(const void* in, int n_img, int h, int w, int in_cstride, int in_coff, int cin,
                             const void* weights, int cout, const float* bias, int flags, void* out, int out_cstride,
                             int out_coff, const void* mask, int mask_cstride, int mask_coff, int accumulate, int* err,
                             cudaStream_t s);

// The same, and the 2x2 average pool of the output as a dense [n][h/2][w/2][cout] tensor (pool may be
// null): for 32 dense input channels, bf16 outputs and even h and w.
cudaError_t rfk_unet_conv3x3_pool(const void* in, int n_img, int h, int w, int in_cstride, int in_coff, int cin,
                                  const void* weights, int cout, const float* bias, int flags, void* out, int out_cstride,
                                  int out_coff, const void* mask, int mask_cstride, int mask_coff, int accumulate, void* pool,
                                  int* err, cudaStream_t s);

// dW[cout][9][cin] (f32) += sum over pixels of dY[p][n] * X[p + tap][c], on tcgen05. dy: dY as
// dense NHWC bf16 (cout channels); x: X as NHWC bf16, channels x_coff .. x_coff + cin of
// x_cstride. w must be a multiple of 64, cin and cout of 32.
cudaError_t rfk_unet_wgrad3x3(const void* dy, const void* x, int x_cstride, int x_coff, int n_img, int h, int w, int cout,
                              int cin, float* dw, int* err, cudaStream_t s);
// The same, and db[n] += sum over pixels of dY[p][n] (db may be null).
cudaError_t rfk_unet_wgrad3x3_bias(const void* dy, const void* x, int x_cstride, int x_coff, int n_img, int h, int w, int cout,
                                   int cin, float* dw, float* db, int* err, cudaStream_t s);
// With db in 64 bits: as many partial sums as there are CTAs meet in it.
cudaError_t rfk_unet_wgrad3x3_bias64(const void* dy, const void* x, int x_cstride, int x_coff, int n_img, int h, int w, int cout,
                                     int cin, float* dw, double* db, int* err, cudaStream_t s);

// Network input (32 bf16 channels per pixel) of a float4 histogram rendered at `spp` and its
// tonemapped image `base` (float4).
cudaError_t rfk_unet_features(const float4* bins, const float4* base, size_t npx, float spp, void* out, cudaStream_t s);
// 2x2 average pool of a channel slice into a dense [n][h/2][w/2][c] tensor.
cudaError_t rfk_unet_avgpool(const void* in, int n_img, int h, int w, int cstride, int coff, int c, void* out,
                             cudaStream_t s);
// Gradient through the upsample (2x2 sums of a slice of g) times (cat > 0), the upsampled activation
// in the same slice of the [n][2h][2w] concatenation; out [n][h][w][c].
cudaError_t rfk_unet_up_backward(const void* g, int gcstride, int gcoff, const void* cat, int n_img, int h, int w, int c,
                                 void* out, cudaStream_t s);
// Gradient of a skip slice feeding a concatenation and an average pool, times its ReLU derivative.
cudaError_t rfk_unet_skip_backward(const void* gcat, int cstride, int coff, const void* gpool, const void* cat, int n_img,
                                   int h, int w, int c, void* out, cudaStream_t s);
// Mean squared error of base + output (RFK_UNET_RGBOUT) against f32 RGBA targets;
// bf16 gradient.
cudaError_t rfk_unet_mse(const float4* out, const float4* base, const float4* target, size_t npx, void* grad, double* loss,
                         cudaStream_t s);
// Adam step of all layers, writing the bf16 forward and input-gradient copies.
cudaError_t rfk_unet_adam(const rfk_unet_layer* layers, int n, float lr, float b1, float b2, float eps, int step, cudaStream_t s);
// base + network output to an image (RFK_HALF3 .. RFK_FLOAT4; alpha as the tonemapper's).
cudaError_t rfk_unet_to_image(const float4* net, const float4* base, const float4* bins, size_t npx, void* out, int format,
                              cudaStream_t s);

#ifdef __cplusplus
}
#endif
