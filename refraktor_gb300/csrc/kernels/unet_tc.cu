// Tensor-core kernels of the learned denoiser: 3x3 convolutions (stride 1,
// zero padding 1) of bf16 NHWC activations as implicit GEMMs on tcgen05, with
// f32 accumulators in TMEM.
//
// conv3x3_tc (forward and input-gradient): persistent CTAs walk tiles of R
// image rows x 128 output pixels x BN output channels.
//   D[p, n] = sum over taps t and input channels c of A[p + t, c] * W[n, t, c]
// The K loop runs over input channel blocks of BK and, depending on MODE
// (conv_cfg), over taps, tap rows or neither: the A tile of a K block is a
// TMA box of the NHWC input at the tile's offset - the padding comes from
// TMA's zero fill outside the image - and the B tiles boxes (BK x BN) of the
// weights [cout][9][cin]. A producer warp (one lane) issues the TMA loads into
// a ring of shared-memory stages, an MMA warp issues tcgen05.mma
// (M 128, N BN, K 16 per instruction) and frees each stage with
// tcgen05.commit; eight epilogue warps read the accumulator rows from TMEM
// (two per lane quarter) and apply the epilogue: bias, ReLU, a
// ReLU-derivative mask, then bf16 rows by TMA store, or f32 or accumulating
// stores. conv3x3_walk streams pixel pairs through layers of 32 input channels.
// The input gradient of a conv is the same kernel on the output gradient with
// the weights transposed and the taps flipped ([cin][9][cout]).
//
// wgrad3x3_rows and wgrad3x3_cols (weight gradient): dW[n, t, c] = sum over
// pixels p of dY[p, n] * X[p + t, c], GEMMs with K = pixels (64 of an image row at
// a time, W a multiple of 64), M = output channels, and stacked on them tap rows
// where they are few, N = input channels times the three column taps. Both
// operands are read MN-major straight from NHWC; a column tap is the same box
// from one pixel line further on, a tap row another row of dY (zero fill outside
// the image). CTAs split K and add their partial sums into dW (f32) atomically.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "tc_ptx.cuh"
#include "unet_kernels.h"

namespace {

using bf16 = __nv_bfloat16;

// ------------------------------------------------------------------ conv ----
struct conv_args {
    int n_img, h, w, tiles_x;
    int cin, cin_off;  // K channels and their offset in the input tensor
    int cout;
    void* out;
    int out_cstride, out_coff;
    const float* bias;
    int relu;
    int out_f32;  // store f32 instead of bf16
    int out_rgb;  // f32: the first four channels only
    int up2;      // store at the 2x2 pixels of a (2h, 2w) output
    const bf16* mask;
    int mask_cstride, mask_coff;
    int accumulate;
    int tma_out;  // bf16 output through shared memory and TMA stores
    int band;     // conv3x3_walk: output rows per task
    bf16* pool;   // conv3x3_walk: the output's 2x2 average pool too, dense (null: not wanted)
    int* err;
};

// Tap reuse. MODE 0: one K block per (tap, input channel block), its A box
// the 128 pixels of each tile row shifted by the tap. MODE 1 (column taps): a
// K block covers one tap row dy and the three column taps; its A box holds
// 136 pixels of each image row from x0 - 1 on (130 used; 136 keeps every row
// 1024-byte aligned for 128-byte swizzle and 512-byte aligned for 64-byte
// swizzle) and the MMAs of column tap dx read it through a descriptor that
// starts dx pixel lines later. MODE 2 (all taps): a K block covers all nine
// taps of one input channel block; its A box holds the tile's R rows plus the
// row above and below (R + 2 rows of 136 pixels) and the MMAs of tap (dy, dx)
// start at row r + dy, pixel line dx; the layer's weights (up to three input
// channel blocks x nine taps, one output tile) are loaded once per CTA and
// stay in shared memory, so the stages carry only the input. The input
// crosses L2 nine, three or (R + 2) / R times per layer.
template <int BK, int BN, int MODE>
struct conv_cfg {
    // R image rows per tile (R accumulators of 128 x BN): small-N layers move
    // R times the bytes per pipeline stage, so the stage round trip is shared
    // (128 channels: two rows share each weight tile)
    static constexpr int R = BN == 128 ? 2 : BN == 256 ? 1 : 128 / BN;
    static constexpr int A_PIX = MODE ? 136 : 128;                // pixel lines per image row
    static constexpr int A_ROWS = MODE == 2 ? R + 2 : R;           // image rows per A box
    static constexpr uint32_t A_ROW = (uint32_t)A_PIX * BK * 2u;   // one image row segment
    static constexpr uint32_t A_BYTES = A_ROWS * A_ROW;
    static constexpr int NT = MODE == 2 ? 9 : (MODE == 1 ? 3 : 1);  // taps per K block
    static constexpr int NB = MODE == 2 ? 0 : NT;                    // weight tiles per stage
    static constexpr uint32_t B_TILE = (uint32_t)BN * BK * 2u;
    static constexpr int KB_RES = 3;                                 // resident input channel blocks (MODE 2)
    static constexpr uint32_t B_RES = MODE == 2 ? KB_RES * 9u * B_TILE : 0u;
    static constexpr uint32_t LOAD_BYTES = A_BYTES + NB * B_TILE;  // bytes the TMA writes per stage
    static constexpr uint32_t STAGE_BYTES = (LOAD_BYTES + 1023u) & ~1023u;
    static constexpr int TAPS = MODE == 2 ? 1 : (MODE == 1 ? 3 : 9);  // K blocks per input channel block
    // output staging: two tiles of 128 pixels x OC channels
    static constexpr int OC = BN % 64 == 0 ? 64 : 32;
    static constexpr uint32_t OUT_TILE = 128u * OC * 2u;
    // one persistent CTA per SM: as many stages as fit in 224 KB with the weights and
    // the output tiles, at most 8
    static constexpr uint32_t BUDGET = 229376u - 2u * OUT_TILE;
    static constexpr int STAGES = ((BUDGET - B_RES) / STAGE_BYTES > 8) ? 8 : (int)((BUDGET - B_RES) / STAGE_BYTES);
    static constexpr uint32_t SMEM = B_RES + STAGES * STAGE_BYTES + 2u * OUT_TILE + 1024u;
    static constexpr uint32_t TMEM_COLS = 2u * R * BN;  // two sets of R accumulators
    static_assert(MODE == 0 || (A_ROW % 512u == 0 && A_BYTES % 1024u == 0 && B_TILE % 1024u == 0 && B_RES % 1024u == 0),
                  "tap-reuse tiles must stay swizzle-aligned");
    static_assert(STAGES >= 2, "at least two stages");
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void store_bf16x16(bf16* dst, const float (&v)[16]) {
    uint4* d = reinterpret_cast<uint4*>(dst);
#pragma unroll
    for (int q = 0; q < 2; q++) {
        __nv_bfloat162 h[4];
#pragma unroll
        for (int j = 0; j < 4; j++) h[j] = __floats2bfloat162_rn(v[8 * q + 2 * j], v[8 * q + 2 * j + 1]);
        d[q] = *reinterpret_cast<uint4*>(h);
    }
}

__device__ __forceinline__ void load_bf16x16(const bf16* src, float (&v)[16]) {
    const uint4* s = reinterpret_cast<const uint4*>(src);
#pragma unroll
    for (int q = 0; q < 2; q++) {
        uint4 u = s[q];
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            float2 f = __bfloat1622float2(h[j]);
            v[8 * q + 2 * j] = f.x;
            v[8 * q + 2 * j + 1] = f.y;
        }
    }
}

constexpr int kEpiWarps = 8;  // two warps per TMEM lane quarter, each half of the columns

// Bias; ReLU and ReLU-derivative mask of N consecutive output channels of one pixel.
template <int N>
__device__ __forceinline__ void conv_bias(const conv_args& p, float (&v)[N], int ch) {
    if (!p.bias) return;
    const float4* bb = reinterpret_cast<const float4*>(p.bias + ch);
#pragma unroll
    for (int q = 0; q < N / 4; q++) {
        const float4 f = __ldg(bb + q);
        v[4 * q] += f.x;
        v[4 * q + 1] += f.y;
        v[4 * q + 2] += f.z;
        v[4 * q + 3] += f.w;
    }
}
template <int N>
__device__ __forceinline__ void conv_activate(const conv_args& p, float (&v)[N], int ch, size_t pix, bool valid) {
    if (p.relu) {
#pragma unroll
        for (int j = 0; j < N; j++) v[j] = fmaxf(v[j], 0.0f);
    }
    if (p.mask && valid) {
#pragma unroll
        for (int g = 0; g < N; g += 16) {
            float m[16];
            load_bf16x16(p.mask + pix * p.mask_cstride + p.mask_coff + ch + g, m);
#pragma unroll
            for (int j = 0; j < 16; j++) v[g + j] = m[j] > 0.0f ? v[g + j] : 0.0f;
        }
    }
}

// f32 and accumulating outputs: a lane stores its pixel's N channels from ch on.
template <int N>
__device__ __forceinline__ void store_direct(const conv_args& p, float (&v)[N], size_t pix, int ch) {
    if (p.out_rgb) {
        if (ch == 0) static_cast<float4*>(p.out)[pix] = make_float4(v[0], v[1], v[2], v[3]);
        return;
    }
    const size_t at = pix * p.out_cstride + p.out_coff + ch;
    if (p.out_f32) {
        float4* dst = reinterpret_cast<float4*>(static_cast<float*>(p.out) + at);
#pragma unroll
        for (int q = 0; q < N / 4; q++) {
            const float4 o = p.accumulate ? dst[q] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            dst[q] = make_float4(v[4 * q] + o.x, v[4 * q + 1] + o.y, v[4 * q + 2] + o.z, v[4 * q + 3] + o.w);
        }
        return;
    }
#pragma unroll
    for (int g = 0; g < N; g += 16) {
        bf16* dst = static_cast<bf16*>(p.out) + at + g;
        float o[16];
        load_bf16x16(dst, o);
#pragma unroll
        for (int j = 0; j < 16; j++) o[j] += v[g + j];
        store_bf16x16(dst, o);
    }
}

// N channels of pixel px, from channel c0 of a tile of 128 pixels x OC
// channels in shared memory, swizzled as the output's tensor map has it
// (128- or 64-byte rows), so that the lanes' 16-byte writes meet no bank twice.
template <int OC, int N>
__device__ __forceinline__ void stage_bf16(uint8_t* tile, int px, int c0, const float (&v)[N]) {
#pragma unroll
    for (int q = 0; q < N / 8; q++) {
        __nv_bfloat162 hh[4];
#pragma unroll
        for (int j = 0; j < 4; j++) hh[j] = __floats2bfloat162_rn(v[8 * q + 2 * j], v[8 * q + 2 * j + 1]);
        const uint32_t k = (uint32_t)(c0 / 8 + q);  // 16-byte piece of the pixel
        const uint32_t sw = OC == 64 ? (k ^ ((uint32_t)px & 7u)) : (k ^ (((uint32_t)px >> 1) & 3u));
        *reinterpret_cast<uint4*>(tile + px * (OC * 2) + sw * 16) = *reinterpret_cast<uint4*>(hh);
    }
}

// One thread: the staged tile to channels ch .. of pixels xt * 128 .. of a row
// (with up2 to the 2 x 2 pixels of each).
__device__ __forceinline__ void store_row(const conv_args& p, const CUtensorMap* map, const uint8_t* tile, int ch, int xt, int row) {
    if (p.up2) {
#pragma unroll
        for (int d = 0; d < 4; d++) tc::tma_store_5d(map, tile, ch, d & 1, xt * 128, d >> 1, row);
    } else {
        tc::tma_store_3d(map, tile, ch, xt * 128, row);
    }
    tc::tma_store_commit();
}

// Drains R accumulator rows of 128 x BN (TMEM columns from acc on) into the
// output: image rows y0 + r, pixels xt * 128 ..; warp (quarter, half) reads
// TMEM lanes 32 quarter .. 32 quarter + 31 = pixels, columns of its half.
// f32 and accumulating outputs: each lane stores its pixel's channels.
template <int R, int BN>
__device__ __forceinline__ void conv_epilogue(const conv_args& p, uint32_t acc, int img, int y0, int xt, int n0, int quarter,
                                              int half, int lane) {
    const int x = xt * 128 + quarter * 32 + lane;
#pragma unroll 1
    for (int r = 0; r < R; r++) {
        const int y = y0 + r;
        const bool valid = x < p.w && y < p.h;
        const size_t pix = ((size_t)img * p.h + (valid ? y : 0)) * p.w + (valid ? x : 0);
#pragma unroll 1
        for (int c = half * (BN / 2); c < (half + 1) * (BN / 2); c += 16) {
            if (p.out_rgb && n0 + c) break;
            float v[16];
            tc::tmem_ld16(acc + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(r * BN + c), v);
            if (!valid) continue;
            conv_bias<16>(p, v, n0 + c);
            conv_activate<16>(p, v, n0 + c, pix, true);
            store_direct<16>(p, v, pix, n0 + c);
        }
    }
}

// As conv_epilogue, for bf16 outputs: a row's 128 pixels x OC channels are
// assembled in shared memory and leave as one TMA store, or four with up2. A lane storing its own
// pixel's 32-byte pieces touches 32 lines per instruction: for a 1080p image the
// 64-channel layer with up2 took 141 us that way and takes 66, the 128-channel one
// 88 and 45, a plain 32 -> 64 layer 47 and 39.
// Two staging tiles; `flip` counts the tiles written so far.
template <int R, int BN, int OC>
__device__ __forceinline__ void conv_epilogue_tma(const conv_args& p, const CUtensorMap* map, uint8_t* outbuf, uint32_t acc, int img,
                                                  int y0, int xt, int n0, int quarter, int half, int lane, uint32_t& flip) {
    constexpr int W = OC / 2;  // channels of a warp's half
    const int px = quarter * 32 + lane, x = xt * 128 + px;
    const bool leader = threadIdx.x == 0;
#pragma unroll 1
    for (int r = 0; r < R && y0 + r < p.h; r++) {
        const int y = y0 + r;
        const bool valid = x < p.w;
        const size_t pix = ((size_t)img * p.h + y) * p.w + (valid ? x : 0);
#pragma unroll 1
        for (int c = 0; c < BN; c += OC, flip++) {
            float v[W];
            const uint32_t at = acc + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(r * BN + c + half * W);
            if constexpr (W == 32) tc::tmem_ld32(at, v);
            else tc::tmem_ld16(at, v);
            conv_bias<W>(p, v, n0 + c + half * W);
            conv_activate<W>(p, v, n0 + c + half * W, pix, valid);
            uint8_t* tile = outbuf + (flip & 1u) * (128u * OC * 2u);
            // the tile's previous store has read it
            if (leader) tc::tma_store_wait_read<1>();
            tc::named_barrier(1, 32 * kEpiWarps);
            stage_bf16<OC, W>(tile, px, half * W, v);
            tc::fence_async();
            tc::named_barrier(2, 32 * kEpiWarps);
            if (leader) store_row(p, map, tile, p.out_coff + n0 + c, xt, img * p.h + y);
        }
    }
}

// Persistent: one CTA per SM walks the tiles (R rows x 128-pixel segment x BN
// output channels) t = blockIdx.x, blockIdx.x + gridDim.x, ...
// Warps 0-7: epilogue (warp w reads TMEM lane quarter w % 4, column half
// w / 4), warp 8 lane 0: TMA producer over a ring of stages that runs across
// tiles, warp 9: MMA issuer (the whole warp, see tc::mma_bf16). Two TMEM
// accumulators: the MMAs of tile i + 1 run while the epilogue drains tile i
// (acc_full / acc_empty barriers).
template <int BK, int BN, int MODE>
__global__ void __launch_bounds__(320, 1) conv3x3_tc(const __grid_constant__ CUtensorMap tmA,
                                                     const __grid_constant__ CUtensorMap tmB,
                                                     const __grid_constant__ CUtensorMap tmO, conv_args p) {
    using C = conv_cfg<BK, BN, MODE>;
    extern __shared__ uint8_t smem_dyn[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[C::STAGES], empty[C::STAGES], acc_full[2], acc_empty[2], wbar;
    __shared__ uint32_t tmem_base;
    __shared__ int s_fail;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    uint8_t* const res = base;                   // resident weights (MODE 2)
    uint8_t* const stages = base + C::B_RES;
    uint8_t* const outbuf = stages + C::STAGES * C::STAGE_BYTES;

    const int ntn = p.cout / BN;                           // N tiles
    const int rows_t = (p.h + C::R - 1) / C::R;            // row groups per image
    const int ntiles = p.n_img * rows_t * p.tiles_x * ntn;
    const int kpt = p.cin / BK;                            // K blocks per tap
    const int nk = C::TAPS * kpt;

    if (warp == 0) tc::tmem_alloc(&tmem_base, C::TMEM_COLS);
    if (threadIdx.x == 32) {
        for (int s = 0; s < C::STAGES; s++) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            tc::mbar_init(&acc_full[b], 1);
            tc::mbar_init(&acc_empty[b], kEpiWarps);  // one arrival per epilogue warp
        }
        tc::mbar_init(&wbar, 1);
        s_fail = 0;
        tc::mbar_fence_init();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);

    if (warp == kEpiWarps) {
        if (lane == 0) {
            // producer: the stage ring runs across tiles
            uint32_t g = 0;
            bool ok = true;
            if (MODE == 2) {
                // the layer's weights (one output tile: cout == BN), all taps and input blocks
                tc::mbar_expect_tx(&wbar, (uint32_t)kpt * 9u * C::B_TILE);
                for (int cb = 0; cb < kpt; cb++)
#pragma unroll
                    for (int t9 = 0; t9 < 9; t9++)
                        tc::tma_load_2d(res + (cb * 9 + t9) * C::B_TILE, &tmB, &wbar, t9 * p.cin + cb * BK, 0);
            }
            for (int t = blockIdx.x; ok && t < ntiles; t += gridDim.x) {
                const int mt = t / ntn, n0 = (t - mt * ntn) * BN;
                const int xt = mt % p.tiles_x;
                const int y = ((mt / p.tiles_x) % rows_t) * C::R;
                const int img = mt / (p.tiles_x * rows_t);
                for (int kb = 0; kb < nk; kb++, g++) {
                    const uint32_t s = g % C::STAGES, r = g / C::STAGES;
                    if (r > 0 && !tc::mbar_wait(&empty[s], (r - 1) & 1)) {
                        ok = false;
                        break;
                    }
                    const int tap = kb / kpt, cb = kb - tap * kpt;
                    uint8_t* sa = stages + (size_t)s * C::STAGE_BYTES;
                    tc::mbar_expect_tx(&full[s], C::LOAD_BYTES);
                    if (MODE == 2) {
                        // rows y - 1 .. y + R, pixels x0 - 1 .. x0 + 134 (weights resident)
                        tc::tma_load_4d(sa, &tmA, &full[s], p.cin_off + cb * BK, xt * 128 - 1, y - 1, img);
                    } else if (MODE == 1) {
                        // tap = dy row: pixels x0 - 1 .. x0 + 134, the three column taps' weights
                        tc::tma_load_4d(sa, &tmA, &full[s], p.cin_off + cb * BK, xt * 128 - 1, y + tap - 1, img);
#pragma unroll
                        for (int dx = 0; dx < 3; dx++)
                            tc::tma_load_2d(sa + C::A_BYTES + dx * C::B_TILE, &tmB, &full[s], (tap * 3 + dx) * p.cin + cb * BK,
                                            n0);
                    } else {
                        tc::tma_load_4d(sa, &tmA, &full[s], p.cin_off + cb * BK, xt * 128 + tap % 3 - 1, y + tap / 3 - 1,
                                        img);
                        tc::tma_load_2d(sa + C::A_BYTES, &tmB, &full[s], tap * p.cin + cb * BK, n0);
                    }
                }
            }
            if (!ok) {
                atomicExch(&s_fail, 1);
                // let the copies in flight land before the CTA exits (bounded)
                for (uint32_t q = g >= (uint32_t)C::STAGES ? g - C::STAGES : 0; q < g; q++)
                    tc::mbar_wait(&full[q % C::STAGES], (q / C::STAGES) & 1);
            }
            if (MODE == 2 && !tc::mbar_wait(&wbar, 0)) atomicExch(&s_fail, 1);
        }
    } else if (warp == kEpiWarps + 1) {
        // the whole warp, see tc::mma_bf16
        const uint32_t one = lane == 0;
        {
            constexpr uint32_t idesc = tc::idesc_bf16(128, BN), HI = tc::desc_hi(BK * 2);
            uint32_t g = 0;
            bool ok = MODE != 2 || tc::all_lanes(tc::mbar_wait(&wbar, 0));
            const uint32_t sres = tc::smem_u32(res);
            int i = 0;
            for (int t = blockIdx.x; ok && t < ntiles; t += gridDim.x, i++) {
                const int b = i & 1;
                if (i >= 2 && !tc::all_lanes(tc::mbar_wait(&acc_empty[b], ((i >> 1) - 1) & 1))) {
                    ok = false;
                    break;
                }
                tc::fence_after();
                const uint32_t acc = tmem + (uint32_t)(b * C::R * BN);
                for (int kb = 0; kb < nk; kb++, g++) {
                    const uint32_t s = g % C::STAGES;
                    if (!tc::all_lanes(tc::mbar_wait(&full[s], (g / C::STAGES) & 1))) {
                        ok = false;
                        break;
                    }
                    tc::fence_after();
                    const uint32_t sa = tc::smem_u32(stages + (size_t)s * C::STAGE_BYTES);
                    // MODE 2: the resident weights of input block kb, else the stage's
                    const uint32_t sb = MODE == 2 ? sres + (uint32_t)(kb * 9) * C::B_TILE : sa + C::A_BYTES;
                    // descriptors of the stage's first tiles; the others differ only in the
                    // start address field (bits 0-13, 16-byte units; shared memory < 256 KB,
                    // so adding the compile-time offset cannot carry out of it)
                    const uint32_t a0 = tc::desc_lo(sa), b0 = tc::desc_lo(sb);
#pragma unroll
                    for (int r = 0; r < C::R; r++)
#pragma unroll
                        for (int t = 0; t < C::NT; t++) {
                            // MODE 2: tap t = (dy, dx) reads row r + dy; MODE 1: t = dx
                            const int dy = MODE == 2 ? t / 3 : 0, dx = MODE == 2 ? t % 3 : t;
#pragma unroll
                            for (int kk = 0; kk < BK / 16; kk++)
                                tc::mma_bf16<HI, HI>(one, acc + (uint32_t)(r * BN),
                                                     a0 + (uint32_t)(((r + dy) * C::A_ROW + dx * (BK * 2) + kk * 32) >> 4),
                                                     b0 + (uint32_t)((t * C::B_TILE + kk * 32) >> 4), idesc,
                                                     (kb | t | kk) != 0 ? 1u : 0u);
                        }
                    tc::mma_commit(one, &empty[s]);
                }
                tc::mma_commit(one, &acc_full[b]);  // also on failure: arrives once the issued MMAs are done
            }
            if (!ok) atomicExch(&s_fail, 1);
        }
    } else {
        // epilogue: warps 0-7; TMEM lane 32 * (warp % 4) + lane = tile row,
        // columns [half * BN / 2, (half + 1) * BN / 2)
        const int quarter = warp & 3, half = warp >> 2;
        uint32_t flip = 0;
        int i = 0;
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x, i++) {
            const int b = i & 1;
            // all epilogue warps go on or stop together (they meet at barriers below)
            const bool got = tc::named_barrier_all(1, 32 * kEpiWarps, tc::all_lanes(tc::mbar_wait(&acc_full[b], (i >> 1) & 1)));
            if (!got) {
                if (lane == 0) atomicExch(&s_fail, 1);
                break;
            }
            tc::fence_after();
            const int mt = t / ntn, n0 = (t - mt * ntn) * BN;
            const int xt = mt % p.tiles_x;
            const int y0 = ((mt / p.tiles_x) % rows_t) * C::R;
            const int img = mt / (p.tiles_x * rows_t);
            if (p.tma_out)
                conv_epilogue_tma<C::R, BN, C::OC>(p, &tmO, outbuf, tmem + (uint32_t)(b * C::R * BN), img, y0, xt, n0, quarter, half,
                                                   lane, flip);
            else
                conv_epilogue<C::R, BN>(p, tmem + (uint32_t)(b * C::R * BN), img, y0, xt, n0, quarter, half, lane);
            // the accumulator may be overwritten once all epilogue warps have read it
            tc::fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[b]);
        }
        if (threadIdx.x == 0) tc::tma_store_wait<0>();
    }
    tc::fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && s_fail) atomicExch(p.err, 1);
    if (warp == 0) tc::tmem_dealloc(tmem, C::TMEM_COLS);
}

// conv3x3_walk: 32 dense input channels, tiles of 32 output channels.
struct walk_cfg {
    static constexpr uint32_t A_ROW = 136u * 128u;  // 136 pixel pairs of an input row, from x0 - 2 on
    static constexpr uint32_t B_TILE = 32u * 64u, RES = 9u * B_TILE;
    static constexpr int SLOTS = 4;                 // accumulators of 128 x 32 per strip and pixel of a pair
    static constexpr int DONE = 16;                 // barriers of a strip's input rows
    static constexpr int STAGES = 7;
    static constexpr uint32_t OUT_TILE = 128u * 64u * 2u;  // two per strip
    static constexpr uint32_t SMEM = RES + STAGES * A_ROW + 4u * OUT_TILE + 1024u;
};

// Row-streaming convolution of 32 input channels whose sums keep the order of
// conv3x3_tc's, tap after tap. A 32-channel layer moves 64 bytes per pixel each way,
// and TMA boxes of 64-byte rows get half the memory rate of 128-byte ones, so the
// tensors are taken as images of w / 2 pixel pairs with 64 channels: M is 128 pairs,
// the left and the right pixels have accumulators of their own, and a column tap
// reads the half line (the right one of the pair before, both of the pair, the left
// one of the pair after) that holds its pixel. (One accumulator for both pixels and
// weights of 0 for the pixels that a tap row does not reach make 8 MMAs of N 192 of
// the 12 of N 96, 109 us instead of 130, but 0 times an infinity is not 0.)
// An MMA is bound by its A tile (M 128 x K 16 takes 45 cycles at N 32 and 56 at N 96),
// so the three tap rows lie in N, and they meet in one accumulator per output row:
// input row i is tap row 2 of output row i - 2, tap row 1 of i - 1 and tap row 0 of i,
// whose accumulators are neighbours in a ring of four (96
// columns; 32 or 64 at a band's ends, in two parts at the ring's). MMAs of different
// input rows overlap in accumulators but not in their base, which no rule orders: the
// next row of a strip is issued when the one before is done. Two strips in turn, each
// with accumulator rings and an epilogue group of its own, hide that wait in part.
// The epilogue clears an accumulator that it has read.
// 16 images of 512 x 512, 32 -> 32 channels: 130 us, conv3x3_tc 138; with a mask 179
// and 289; 32 -> 96: 369 and 423.
__global__ void __launch_bounds__(320, 1) conv3x3_walk(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                                                       const __grid_constant__ CUtensorMap tmO, conv_args p) {
    using C = walk_cfg;
    extern __shared__ uint8_t smem_dyn[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[C::STAGES], empty[C::STAGES], done[2][C::DONE], slot_empty[2][C::SLOTS], wbar;
    __shared__ uint32_t tmem_base;
    __shared__ int s_fail;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    uint8_t* const res = base;
    uint8_t* const outbuf = base + C::RES;
    uint8_t* const stages = outbuf + 4 * C::OUT_TILE;
    // this CTA's 32 output channels, and its tasks (bands of columns of 128 pairs)
    // among those of the CTAs that share them; strip k takes every other one
    const int ntn = p.cout / 32, n0 = ((int)blockIdx.x % ntn) * 32;
    const int bands = (p.h + p.band - 1) / p.band;
    const int ntasks = p.n_img * bands * p.tiles_x, first = (int)blockIdx.x / ntn;
    const int step = ((int)gridDim.x - (int)blockIdx.x % ntn + ntn - 1) / ntn;

    if (warp == 0) tc::tmem_alloc(&tmem_base, 512u);
    if (threadIdx.x == 32) {
        for (int s = 0; s < C::STAGES; s++) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        for (int k = 0; k < 2; k++) {
            for (int s = 0; s < C::DONE; s++) tc::mbar_init(&done[k][s], 1);
            for (int s = 0; s < C::SLOTS; s++) tc::mbar_init(&slot_empty[k][s], 4);
        }
        tc::mbar_init(&wbar, 1);
        s_fail = 0;
        tc::mbar_fence_init();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
    if (warp < 8)
        for (int c = 0; c < C::SLOTS; c++)
            for (int a = 0; a < 64; a += 32)
                tc::tmem_zero32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * 256 + c * 64 + a));
    tc::fence_before();
    __syncthreads();
    tc::fence_after();

    // The producer and the issuing warp go through the strips' input rows in the
    // same order: one row of each strip that has rows left, in turn.
    struct strip {
        int t, i, rows;  // task, input row in it, its output rows
    };
    auto open = [&](strip& q, int t) {
        q.t = t;
        q.i = 0;
        q.rows = t < ntasks ? min(p.band, p.h - ((t / p.tiles_x) % bands) * p.band) : 0;
    };

    if (warp == 8) {
        if (lane == 0) {
            tc::mbar_expect_tx(&wbar, C::RES);
            for (int dx = 0; dx < 3; dx++)
                for (int dy = 0; dy < 3; dy++)  // stacked as [dy 2 | dy 1 | dy 0]
                    tc::tma_load_2d(res + (uint32_t)(dx * 3 + 2 - dy) * C::B_TILE, &tmB, &wbar, (dy * 3 + dx) * 32, n0);
            int issued = 0;
            bool ok = true;
            strip st[2];
            open(st[0], first);
            open(st[1], first + step);
            while (ok && (st[0].t < ntasks || st[1].t < ntasks)) {
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    strip& q = st[k];
                    if (!ok || q.t >= ntasks) continue;
                    const int s = issued % C::STAGES, round = issued / C::STAGES;
                    if (round > 0 && !tc::mbar_wait(&empty[s], (round - 1) & 1)) {
                        ok = false;
                        continue;
                    }
                    const int y0 = ((q.t / p.tiles_x) % bands) * p.band;
                    tc::mbar_expect_tx(&full[s], C::A_ROW);
                    tc::tma_load_4d(stages + (uint32_t)s * C::A_ROW, &tmA, &full[s], 0, q.t % p.tiles_x * 128 - 1,
                                    y0 + q.i - 1, q.t / (p.tiles_x * bands));
                    issued++;
                    if (++q.i == q.rows + 2) open(q, q.t + 2 * step);
                }
            }
            if (!ok) {
                atomicExch(&s_fail, 1);
                // let the copies in flight land before the CTA exits (bounded)
                for (int q = issued >= C::STAGES ? issued - C::STAGES : 0; q < issued; q++)
                    tc::mbar_wait(&full[q % C::STAGES], (q / C::STAGES) & 1);
            }
            if (!tc::mbar_wait(&wbar, 0)) atomicExch(&s_fail, 1);
        }
    } else if (warp == 9) {
        const uint32_t one = lane == 0;
        constexpr uint32_t AHI = tc::desc_hi(128), BHI = tc::desc_hi(64);
        const uint32_t b0 = tc::desc_lo(tc::smem_u32(res));
        bool ok = tc::all_lanes(tc::mbar_wait(&wbar, 0));
        int n = 0;                 // stages used
        int in[2] = {0, 0};        // input rows issued of a strip
        int out[2] = {0, 0};       // output rows of its earlier tasks
        strip st[2];
        open(st[0], first);
        open(st[1], first + step);
        while (ok && (st[0].t < ntasks || st[1].t < ntasks)) {
#pragma unroll
            for (int k = 0; k < 2; k++) {
                strip& q = st[k];
                if (!ok || q.t >= ntasks) continue;
                const int s = n % C::STAGES;
                ok = tc::all_lanes(tc::mbar_wait(&full[s], (n / C::STAGES) & 1));
                // the strip's row before this one
                if (ok && in[k] > 0) ok = tc::all_lanes(tc::mbar_wait(&done[k][(in[k] - 1) % C::DONE], ((in[k] - 1) / C::DONE) & 1));
                // the accumulator of output row i, read and cleared
                const int o = out[k] + q.i;
                if (ok && q.i < q.rows && o >= C::SLOTS)
                    ok = tc::all_lanes(tc::mbar_wait(&slot_empty[k][o % C::SLOTS], (o / C::SLOTS - 1) & 1));
                if (ok) {
                    tc::fence_after();
                    const uint32_t a0 = tc::desc_lo(tc::smem_u32(stages + (uint32_t)s * C::A_ROW));
                    // output rows lo .. lo + num - 1, of which `part` up to the ring's end
                    const int lo = max(q.i - 2, 0), num = min(q.i, q.rows - 1) - lo + 1;
                    const int slot = (out[k] + lo) % C::SLOTS, part = min(num, C::SLOTS - slot);
                    const uint32_t b = b0 + (uint32_t)(lo - (q.i - 2)) * (C::B_TILE >> 4);
                    for (int at = 0; at < num; at = at ? num : part) {
                        const int m = at ? num - part : part;
                        const uint32_t acc = tmem + (uint32_t)(k * 256 + (at ? 0 : slot) * 32);
                        const uint32_t idesc = tc::idesc_bf16(128, 0) | ((uint32_t)(m * 32 / 8) << 17);
#pragma unroll
                        for (int a = 0; a < 2; a++)
#pragma unroll
                            for (int dx = 0; dx < 3; dx++)
#pragma unroll
                                for (int kk = 0; kk < 2; kk++)
                                    // half lines from the right one of line 0 on
                                    tc::mma_bf16<AHI, BHI>(one, acc + a * 128u, a0 + (uint32_t)((64 + (a + dx) * 64 + kk * 32) >> 4),
                                                           b + (uint32_t)(((at + dx * 3) * C::B_TILE + kk * 32) >> 4), idesc, 1u);
                    }
                    tc::mma_commit(one, &empty[s]);
                    tc::mma_commit(one, &done[k][in[k] % C::DONE]);
                    n++;
                    in[k]++;
                    if (++q.i == q.rows + 2) {
                        out[k] += q.rows;
                        open(q, q.t + 2 * step);
                    }
                }
            }
        }
        if (!ok) atomicExch(&s_fail, 1);
    } else {
        // epilogue group k: the output rows of strip k. A barrier of `done` is used
        // again 16 input rows later; the issuing warp is 7 output rows ahead at most,
        // which is 15 input rows or fewer as a band has two rows at least.
        const int quarter = warp & 3, k = warp >> 2;
        const bool leader = (threadIdx.x & 127) == 0;
        const int pair = quarter * 32 + lane;
        const bool dense = p.out_cstride == 32;
        const uint32_t lane_acc = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(k * 256);
        int in = 0, out = 0;  // input rows of earlier tasks, output rows so far
        bool ok = true;
        float above[32];      // the pair's sum in an even row, for the pool
        for (int t = first + k * step; ok && t < ntasks; t += 2 * step) {
            const int xt = t % p.tiles_x, y0 = ((t / p.tiles_x) % bands) * p.band, img = t / (p.tiles_x * bands);
            const int rows = min(p.band, p.h - y0);
            const int x = (xt * 128 + pair) * 2;
            const bool valid = x < p.w;  // w is even
            for (int q = 0; q < rows; q++, out++) {
                const int g = in + q + 2;
                ok = tc::named_barrier_all(1 + k, 128, tc::all_lanes(tc::mbar_wait(&done[k][g % C::DONE], (g / C::DONE) & 1)));
                if (!ok) {
                    if (lane == 0) atomicExch(&s_fail, 1);
                    break;
                }
                tc::fence_after();
                float v[2][32];  // the pair's pixels
                const uint32_t acc = lane_acc + (uint32_t)(out % C::SLOTS) * 32u;
#pragma unroll
                for (int a = 0; a < 2; a++) tc::tmem_ld32(acc + a * 128u, v[a]);
#pragma unroll
                for (int a = 0; a < 2; a++) tc::tmem_zero32(acc + a * 128u);
                tc::fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&slot_empty[k][out % C::SLOTS]);
                const int y = y0 + q;
                const size_t pix = ((size_t)img * p.h + y) * p.w + (valid ? x : 0);
                // two staging tiles per strip: the store before last has read this one
                uint8_t* const tile = outbuf + (2 * k + (out & 1)) * C::OUT_TILE;
#pragma unroll
                for (int a = 0; a < 2; a++) {
                    conv_bias<32>(p, v[a], n0);
                    conv_activate<32>(p, v[a], n0, pix + a, valid);
                    if (!p.tma_out) {
                        if (valid) store_direct<32>(p, v[a], pix + a, n0);
                    } else if (dense) {
                        stage_bf16<64, 32>(tile, pair, a * 32, v[a]);
                    } else {
                        stage_bf16<32, 32>(tile + a * (C::OUT_TILE / 2), pair, 0, v[a]);
                    }
                }
                if (p.pool) {
                    // as avgpool_kernel adds the stored values (bands start at even rows);
                    // 1080p: 98 us, 62 and 43 in two passes
#pragma unroll
                    for (int j = 0; j < 32; j += 2) {
                        const float2 l = __bfloat1622float2(__floats2bfloat162_rn(v[0][j], v[0][j + 1]));
                        const float2 r = __bfloat1622float2(__floats2bfloat162_rn(v[1][j], v[1][j + 1]));
                        above[j] = q & 1 ? 0.25f * ((above[j] + l.x) + r.x) : l.x + r.x;
                        above[j + 1] = q & 1 ? 0.25f * ((above[j + 1] + l.y) + r.y) : l.y + r.y;
                    }
                    if ((q & 1) && valid) {
                        bf16* dst = p.pool + (((size_t)img * (p.h / 2) + y / 2) * (p.w / 2) + x / 2) * p.cout + n0;
#pragma unroll
                        for (int g = 0; g < 32; g += 16) store_bf16x16(dst + g, reinterpret_cast<float(&)[16]>(above[g]));
                    }
                }
                if (p.tma_out) {
                    tc::fence_async();
                    if (leader) tc::tma_store_wait_read<0>();
                    tc::named_barrier(1 + k, 128);
                    if (leader) {
                        const int row = img * p.h + y;
                        if (dense) {
                            tc::tma_store_3d(&tmO, tile, 0, xt * 128, row);
                        } else {
#pragma unroll
                            for (int a = 0; a < 2; a++)
                                tc::tma_store_5d(&tmO, tile + a * (C::OUT_TILE / 2), p.out_coff + n0, a, xt * 128, 0, row);
                        }
                        tc::tma_store_commit();
                    }
                }
            }
            in += rows + 2;
        }
        if (leader) tc::tma_store_wait<0>();
    }
    tc::fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && s_fail) atomicExch(p.err, 1);
    if (warp == 0) tc::tmem_dealloc(tmem, 512u);
}

// ----------------------------------------------------------------- wgrad ----
struct wgrad_args {
    int n_img, h, w;
    int cout, cin;
    int x_coff;     // first input channel in the NHWC tensor of X
    int kpc;        // stages (wgrad3x3_rows) or rows (wgrad3x3_cols) of a 64-pixel segment per CTA
    int total;      // all of them
    float* dw;      // [cout][9][cin]
    float* db;      // [cout]: sum of dY, in 32 or 64 bits (both null: not wanted)
    double* db64;
    int vec;        // dw is 16-byte aligned
    int* err;
};

// Adds 32 sums to 32 consecutive weights; `vec`: 16-byte aligned.
__device__ __forceinline__ void wgrad_add(float* dst, const float (&v)[32], int vec) {
    if (vec) {
#pragma unroll
        for (int j = 0; j < 32; j += 4)
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + j), "f"(v[j]), "f"(v[j + 1]), "f"(v[j + 2]),
                         "f"(v[j + 3])
                         : "memory");
    } else {
#pragma unroll
        for (int j = 0; j < 32; j++) atomicAdd(dst + j, v[j]);
    }
}

// Bias gradient on the way: two warps that no MMA or copy needs add up the rows of
// dY while these are in shared memory (those of the first input channel tile), a
// pass over dY of its own less per layer (16 images of 512 x 512: 690 us of the
// 15 layers of a step; the weight gradients take 50 us longer in all).
// A lane adds 16 stages' rows in f32 and those sums in 64 bits, and the CTAs add theirs
// in 64 bits too: hundreds of them meet in a bias. 128 x 512 pixels of 32 channels: an
// error of 3e-10 of sum |dY|; 6e-9 in f32 alone, 1.5e-9 with the pass over dY, whose
// blocks are few there.
// One row of 64 pixels x CO channels as TMA left it (swizzled 64- or 128-byte
// pixel lines), CO / 8 lanes to a pixel, by thread t of 64; acc: this lane's 8 channels.
template <int CO>
__device__ __forceinline__ void bias_row(const uint8_t* row, int t, float (&acc)[8]) {
    constexpr int L = CO / 8, PX = 64 / L;  // lanes per pixel, pixels at a time
    const int c = t % L, px = t / L, sw = c ^ (CO == 64 ? px & 7 : px >> 1 & 3);
#pragma unroll
    for (int i = 0; i < 64 / PX; i++) {
        const uint4 u = *reinterpret_cast<const uint4*>(row + (px + i * PX) * (CO * 2) + sw * 16);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float2 f = __bfloat1622float2(h[j]);
            acc[2 * j] += f.x;
            acc[2 * j + 1] += f.y;
        }
    }
}

constexpr int kBiasStages = 16;  // of f32 sums (4: the folds hold wgrad3x3_cols up, 45 us a step)

__device__ __forceinline__ void bias_fold(float (&acc)[8], double (&sum)[8]) {
#pragma unroll
    for (int j = 0; j < 8; j++) {
        sum[j] += (double)acc[j];
        acc[j] = 0.0f;
    }
}

// The warp's sums of its lanes with the same channels, into channels c0 ..
// min(c0 + CO, cout) - 1.
template <int CO>
__device__ __forceinline__ void bias_add(const wgrad_args& p, int c0, int lane, double (&sum)[8]) {
    constexpr int L = CO / 8;
#pragma unroll
    for (int j = 0; j < 8; j++) {
#pragma unroll
        for (int o = L; o < 32; o *= 2) sum[j] += __shfl_xor_sync(0xffffffffu, sum[j], o);
        const int c = c0 + lane * 8 + j;
        if (lane >= L || c >= p.cout) continue;
        if (p.db64) atomicAdd(p.db64 + c, sum[j]);
        else atomicAdd(p.db + c, (float)sum[j]);
    }
}

// Weight gradient of layers with few channels (CO = 32 or 64 output channels,
// input channel tiles of BN = 32 or 64). A stage holds R image rows of a 64-pixel
// segment: R rows of X, 72 pixels from x0 - 1 on, and R + 2 rows of dY, one TMA box
// each. All nine taps read them from there: the three tap rows are dY rows r,
// r + 1 and r + 2 of the stage against X row r (sum_y dY[y] X[y + dy] =
// sum_y' dY[y' - dy] X[y']), stacked in M; the three column taps are N groups
// that start one pixel line after another. With a box for each tap's rows and
// columns a segment row took 24 KB (32 -> 32 channels) or 96 KB (64 -> 64, a launch
// per tap row), which the L2 delivers at 5.4 TB/s (64-byte rows) or 9.2 TB/s; here
// it is 13 or 26 KB. 16 images of 512 x 512, 32 -> 32: 124 us, before 277; 96 -> 32:
// 246 and 720; 256 x 256, 32 -> 64: 60 and 191; 64 -> 64: 74 and 224; 192 -> 64:
// 169 and 515.
template <int CO, int BN>
struct wgrad_rows_cfg {
    static constexpr int R = 2;
    static constexpr int NB = 3 * BN;  // MMA N
    static constexpr uint32_t A_ROW = CO * 2u, A_GROUP = A_ROW * 64u;
    static constexpr uint32_t B_ROW = BN * 2u, B_GROUP = B_ROW * 72u;
    static constexpr uint32_t A_BYTES = (R + 2) * A_GROUP, STAGE_BYTES = A_BYTES + R * B_GROUP;
    // 32 channels leave room for three CTAs on an SM (128 TMEM columns each), or two
    static constexpr int CTAS = CO == 64 ? 1 : BN == 64 ? 2 : 3;
    static constexpr int STAGES = (int)((225u * 1024u / CTAS - 2048u) / STAGE_BYTES);
    static constexpr uint32_t SMEM = STAGES * STAGE_BYTES + 1024u;
    // CO = 64: tap rows 2 and 1 in one accumulator of 128 rows, 0 in another
    static constexpr int ACCS = CO == 64 ? 2 : 1;
    static constexpr uint32_t ACC_COLS = NB <= 128 ? 128u : 256u;
    static_assert(STAGES >= 2, "a ring");
    static_assert(R * B_GROUP >= A_GROUP, "the unused fourth (CO = 64: second) row group of the last MMA is inside the stage");
};

template <int CO, int BN>
__global__ void __launch_bounds__(128) wgrad3x3_rows(const __grid_constant__ CUtensorMap tmA,
                                                     const __grid_constant__ CUtensorMap tmB, wgrad_args p) {
    using C = wgrad_rows_cfg<CO, BN>;
    extern __shared__ uint8_t smem_dyn[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[C::STAGES], empty[C::STAGES], done;
    __shared__ uint32_t tmem_base;
    __shared__ int s_fail;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

    const int c0 = blockIdx.y * BN;
    const int segs_x = p.w / 64, bands = (p.h + C::R - 1) / C::R;
    const int kb0 = blockIdx.x * p.kpc;
    int nk = p.total - kb0;
    if (nk > p.kpc) nk = p.kpc;
    if (nk < 0) nk = 0;
    const bool bias = (p.db || p.db64) && blockIdx.y == 0;

    if (warp == 0) tc::tmem_alloc(&tmem_base, C::ACCS * C::ACC_COLS);
    if (threadIdx.x == 32) {
        for (int s = 0; s < C::STAGES; s++) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], bias ? 3 : 1);
        }
        tc::mbar_init(&done, 1);
        s_fail = 0;
        tc::mbar_fence_init();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);

    if (warp == 0 && lane == 0) {
        int issued = 0;
        bool ok = true;
        for (int kb = 0; kb < nk; kb++) {
            const int s = kb % C::STAGES, r = kb / C::STAGES;
            if (r > 0 && !tc::mbar_wait(&empty[s], (r - 1) & 1)) {
                ok = false;
                break;
            }
            const int seg = kb0 + kb;
            const int x0 = seg % segs_x * 64;
            const int y0 = seg / segs_x % bands * C::R;
            const int im = seg / (segs_x * bands);
            uint8_t* sa = base + (size_t)s * C::STAGE_BYTES;
            // whole boxes count, zero fill included
            tc::mbar_expect_tx(&full[s], C::STAGE_BYTES);
            tc::tma_load_4d(sa, &tmA, &full[s], 0, x0, y0 - 1, im);
            tc::tma_load_4d(sa + C::A_BYTES, &tmB, &full[s], p.x_coff + c0, x0 - 1, y0, im);
            issued++;
        }
        if (!ok) {
            atomicExch(&s_fail, 1);
            for (int kb = issued - C::STAGES < 0 ? 0 : issued - C::STAGES; kb < issued; kb++)
                tc::mbar_wait(&full[kb % C::STAGES], (kb / C::STAGES) & 1);
        }
    } else if (warp == 1) {
        const uint32_t one = lane == 0;
        constexpr uint32_t idesc = tc::idesc_bf16_bmn(128, C::NB) | (1u << 15);  // A MN-major too
        bool ok = true;
        uint32_t acc = 0;
        for (int kb = 0; kb < nk; kb++) {
            const int s = kb % C::STAGES, r = kb / C::STAGES;
            if (!tc::all_lanes(tc::mbar_wait(&full[s], r & 1))) {
                ok = false;
                break;
            }
            tc::fence_after();
            const uint32_t sa = tc::smem_u32(base + (size_t)s * C::STAGE_BYTES), sb = sa + C::A_BYTES;
            const int rows = min(C::R, p.h - (kb0 + kb) / segs_x % bands * C::R);
            for (int y = 0; y < rows; y++)
#pragma unroll
                for (int kk = 0; kk < 4; kk++) {
                    const uint32_t alo = tc::desc_lo_mn(sa + y * C::A_GROUP + kk * 16 * C::A_ROW, C::A_GROUP);
                    const uint32_t blo = tc::desc_lo_mn(sb + y * C::B_GROUP + kk * 16 * C::B_ROW, C::B_ROW);
                    tc::mma_bf16<tc::desc_hi(C::A_ROW), tc::desc_hi(C::B_ROW)>(one, tmem, alo, blo, idesc, acc);
                    if (C::ACCS == 2)
                        tc::mma_bf16<tc::desc_hi(C::A_ROW), tc::desc_hi(C::B_ROW)>(
                            one, tmem + C::ACC_COLS, tc::desc_lo_mn(sa + (y + 2) * C::A_GROUP + kk * 16 * C::A_ROW, C::A_GROUP),
                            blo, idesc, acc);
                    acc = 1;
                }
            tc::mma_commit(one, &empty[s]);
        }
        tc::mma_commit(one, &done);
        if (!ok) atomicExch(&s_fail, 1);
    } else if (warp >= 2 && bias) {
        const int t = threadIdx.x - 64;
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        double sum[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int kb = 0; kb < nk; kb++) {
            const int s = kb % C::STAGES, r = kb / C::STAGES;
            if (!tc::all_lanes(tc::mbar_wait(&full[s], r & 1))) {
                if (lane == 0) atomicExch(&s_fail, 1);
                break;
            }
            const uint8_t* sa = base + (size_t)s * C::STAGE_BYTES;
            for (int y = 1; y <= C::R; y++) bias_row<CO>(sa + y * C::A_GROUP, t, acc);  // rows past the image are zero
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
            if (kb % kBiasStages == kBiasStages - 1) bias_fold(acc, sum);
        }
        __syncwarp();
        bias_fold(acc, sum);
        bias_add<CO>(p, 0, lane, sum);
    }
    __syncwarp();

    bool got = tc::mbar_wait(&done, 0);
    got = __all_sync(0xffffffffu, got);
    tc::fence_after();
    // accumulator row m: output channel m % CO of dY row m / CO of its MMA, tap
    // row 2 - that; columns [xi BN, (xi + 1) BN) are column tap xi
    if (got && nk > 0) {
#pragma unroll 1
        for (int a = 0; a < C::ACCS; a++) {
            const int g = a * 2 + warp * 32 / CO;
            if (g > 2) break;
            const int m = warp * 32 % CO + lane;
#pragma unroll 1
            for (int c = 0; c < C::NB; c += 32) {
                float v[32];
                tc::tmem_ld32(tmem + a * C::ACC_COLS + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
                wgrad_add(p.dw + ((size_t)m * 9 + (2 - g) * 3 + c / BN) * p.cin + c0 + c % BN, v, p.vec);
            }
        }
    }
    tc::fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && (!got || s_fail)) atomicExch(p.err, 1);
    if (warp == 0) tc::tmem_dealloc(tmem, C::ACCS * C::ACC_COLS);
}

// Weight gradient of layers with 128 output channels or a multiple, in tiles of
// 128 x 32 channels and all nine taps: three accumulators (one per tap row) of 96
// columns (column taps as in wgrad3x3_rows). A CTA walks down the rows of 64-pixel
// columns of the images; the ring holds a row of dY and of X per stage, and a row
// of dY stays for the three rows of X that meet it, so both tensors cross L2 once
// per tile: 21 KB a row against 12 MMAs of 56 cycles, which bound it.
// Boxes for each tap read dY nine times and X three times. 16 images of
// 128 x 128, 64 -> 128: 68 us, before 150; 128 -> 128: 99 and 203; 384 -> 128: 228
// and 436; 64 x 64, 128 -> 256: 64 and 131; 256 -> 256: 103 and 193. (For 64 output
// channels or fewer wgrad3x3_rows fills M with tap rows.)
struct wgrad_cols_cfg {
    static constexpr int BN = 32, NB = 96;
    static constexpr uint32_t A_GROUP = 64u * 128u, A_BYTES = 2u * A_GROUP, B_BYTES = 72u * 64u;
    static constexpr uint32_t STAGE_BYTES = A_BYTES + 5u * 1024u;  // 1024-byte aligned stages
    static constexpr int STAGES = 10;
    static constexpr uint32_t SMEM = STAGES * STAGE_BYTES + 1024u;
};

__global__ void __launch_bounds__(128) wgrad3x3_cols(const __grid_constant__ CUtensorMap tmA,
                                                     const __grid_constant__ CUtensorMap tmB, wgrad_args p) {
    using C = wgrad_cols_cfg;
    extern __shared__ uint8_t smem_dyn[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[C::STAGES], empty[C::STAGES], done;
    __shared__ uint32_t tmem_base;
    __shared__ int s_fail;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

    const int ntiles = p.cin / C::BN;
    const int m0 = (int)(blockIdx.y / ntiles) * 128, c0 = (int)(blockIdx.y % ntiles) * C::BN;
    const int segs_x = p.w / 64;
    // rows of this CTA, counted down the columns one after another
    const int row0 = blockIdx.x * p.kpc, row1 = min(row0 + p.kpc, p.total);
    const bool bias = (p.db || p.db64) && c0 == 0;

    if (warp == 0) tc::tmem_alloc(&tmem_base, 512u);
    if (threadIdx.x == 32) {
        for (int s = 0; s < C::STAGES; s++) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], bias ? 3 : 1);
        }
        tc::mbar_init(&done, 1);
        s_fail = 0;
        tc::mbar_fence_init();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);

    // A run is a CTA's rows within one column. Its stages are the rows from the one
    // above to the one below it, with X only for its own; the MMAs of a row come
    // when the next row's stage is there, and leave the previous row's stage free.
    if (warp == 0 && lane == 0) {
        int k = 0;  // stages issued
        bool ok = true;
        for (int row = row0; ok && row < row1;) {
            const int col = row / p.h, y0 = row % p.h, y1 = min(y0 + row1 - row, p.h);
            const int x0 = col % segs_x * 64, im = col / segs_x;
            for (int y = y0 - 1; y <= y1; y++, k++) {
                const int s = k % C::STAGES, r = k / C::STAGES;
                if (r > 0 && !tc::mbar_wait(&empty[s], (r - 1) & 1)) {
                    ok = false;
                    break;
                }
                const bool own = y >= y0 && y < y1;
                uint8_t* sa = base + (size_t)s * C::STAGE_BYTES;
                tc::mbar_expect_tx(&full[s], C::A_BYTES + (own ? C::B_BYTES : 0u));
                tc::tma_load_4d(sa, &tmA, &full[s], m0, x0, y, im);
                tc::tma_load_4d(sa + C::A_GROUP, &tmA, &full[s], m0 + 64, x0, y, im);
                if (own) tc::tma_load_4d(sa + C::A_BYTES, &tmB, &full[s], p.x_coff + c0, x0 - 1, y, im);
            }
            row += y1 - y0;
        }
        if (!ok) {
            atomicExch(&s_fail, 1);
            for (int j = k - C::STAGES < 0 ? 0 : k - C::STAGES; j < k; j++)
                tc::mbar_wait(&full[j % C::STAGES], (j / C::STAGES) & 1);
        }
    } else if (warp == 1) {
        const uint32_t one = lane == 0;
        constexpr uint32_t idesc = tc::idesc_bf16_bmn(128, C::NB) | (1u << 15);  // A MN-major too
        const uint32_t ring = tc::smem_u32(base);
        bool ok = true;
        uint32_t acc = 0;  // bit d: the accumulator of tap row d holds sums
        int k = 0;         // stage of the run's first row, the one above it
        for (int row = row0; ok && row < row1;) {
            const int y0 = row % p.h, y1 = min(y0 + row1 - row, p.h);
            for (int y = y0; y < y1; y++, k++) {
                // stages k, k + 1, k + 2: dY rows y - 1, y, y + 1
                for (int j = y == y0 ? 0 : 2; ok && j < 3; j++)
                    ok = tc::all_lanes(tc::mbar_wait(&full[(k + j) % C::STAGES], ((k + j) / C::STAGES) & 1));
                if (!ok) break;
                tc::fence_after();
                const uint32_t sb = ring + (uint32_t)((k + 1) % C::STAGES) * C::STAGE_BYTES + C::A_BYTES;
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    // tap row d (X a row lower by d - 1): dY row y - (d - 1)
                    if (y + 1 - d < 0 || y + 1 - d >= p.h) continue;
                    const uint32_t sa = ring + (uint32_t)((k + 2 - d) % C::STAGES) * C::STAGE_BYTES;
#pragma unroll
                    for (int kk = 0; kk < 4; kk++) {
                        tc::mma_bf16<tc::desc_hi(128), tc::desc_hi(64)>(
                            one, tmem + (uint32_t)(d * C::NB), tc::desc_lo_mn(sa + kk * 16 * 128, C::A_GROUP),
                            tc::desc_lo_mn(sb + kk * 16 * 64, 64u), idesc, acc >> d & 1u);
                        acc |= 1u << d;
                    }
                }
                tc::mma_commit(one, &empty[k % C::STAGES]);
            }
            if (!ok) break;
            // the run's last row and the one below it
            tc::mma_commit(one, &empty[k % C::STAGES]);
            tc::mma_commit(one, &empty[(k + 1) % C::STAGES]);
            k += 2;
            row += y1 - y0;
        }
        tc::mma_commit(one, &done);
        if (!ok) atomicExch(&s_fail, 1);
    } else if (warp >= 2 && bias) {
        const int t = threadIdx.x - 64;
        float lo[8] = {0, 0, 0, 0, 0, 0, 0, 0}, hi[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        double lo_sum[8] = {0, 0, 0, 0, 0, 0, 0, 0}, hi_sum[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        bool ok = true;
        int k = 0;
        for (int row = row0; ok && row < row1;) {
            const int y0 = row % p.h, y1 = min(y0 + row1 - row, p.h);
            for (int y = y0 - 1; y <= y1; y++, k++) {
                const int s = k % C::STAGES;
                ok = tc::all_lanes(tc::mbar_wait(&full[s], (k / C::STAGES) & 1));
                if (!ok) break;
                const uint8_t* sa = base + (size_t)s * C::STAGE_BYTES;
                if (y >= y0 && y < y1) {
                    bias_row<64>(sa, t, lo);
                    bias_row<64>(sa + C::A_GROUP, t, hi);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[s]);
                if (k % kBiasStages == kBiasStages - 1) {
                    bias_fold(lo, lo_sum);
                    bias_fold(hi, hi_sum);
                }
            }
            row += y1 - y0;
        }
        if (!ok && lane == 0) atomicExch(&s_fail, 1);
        __syncwarp();
        bias_fold(lo, lo_sum);
        bias_fold(hi, hi_sum);
        bias_add<64>(p, m0, lane, lo_sum);
        bias_add<64>(p, m0 + 64, lane, hi_sum);
    }
    __syncwarp();

    bool got = tc::mbar_wait(&done, 0);
    got = __all_sync(0xffffffffu, got);
    tc::fence_after();
    // accumulator row m of tap row d: output channel m0 + m; columns
    // [32 xi, 32 xi + 32): column tap xi
    const int m = m0 + warp * 32 + lane;
    if (got && row0 < row1 && m < p.cout) {
#pragma unroll 1
        for (int c = 0; c < 3 * C::NB; c += 32) {
            // an only row at the image's edge has met no dY row of this tap row
            const int d = c / C::NB, y = row0 % p.h + 1 - d;
            if (d != 1 && (p.h == 1 || (row1 - row0 == 1 && (y < 0 || y >= p.h)))) continue;
            float v[32];
            tc::tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
            wgrad_add(p.dw + ((size_t)m * 9 + c / 32) * p.cin + c0, v, p.vec);
        }
    }
    tc::fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && (!got || s_fail)) atomicExch(p.err, 1);
    if (warp == 0) tc::tmem_dealloc(tmem, 512u);
}

// ------------------------------------------------------------- tensor maps --
using encode_fn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

encode_fn encoder() {
    static encode_fn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<encode_fn>(p);
    });
    return fn;
}

bool make_map(CUtensorMap* m, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides_bytes,
              const cuuint32_t* box, CUtensorMapSwizzle sw) {
    encode_fn fn = encoder();
    if (!fn) return false;
    cuuint32_t es[5] = {1, 1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base), dims, strides_bytes, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename K>
cudaError_t raise_smem(K kernel, uint32_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

int sm_count_cached() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 1;
    }
    return n;
}

template <int BK, int BN, int MODE>
cudaError_t launch_conv(const CUtensorMap& a, const CUtensorMap& b, const CUtensorMap& o, const conv_args& p, cudaStream_t s) {
    using C = conv_cfg<BK, BN, MODE>;
    static std::once_flag once;
    static cudaError_t attr = cudaSuccess;
    std::call_once(once, [] { attr = raise_smem(conv3x3_tc<BK, BN, MODE>, C::SMEM); });
    if (attr != cudaSuccess) return attr;
    const long long tiles = (long long)p.n_img * ((p.h + C::R - 1) / C::R) * p.tiles_x * (p.cout / BN);
    if (tiles > 0x7FFFFFFFLL) return cudaErrorInvalidValue;
    const int grid = (int)std::min<long long>(tiles, sm_count_cached());
    conv3x3_tc<BK, BN, MODE><<<grid, 32 * (kEpiWarps + 2), C::SMEM, s>>>(a, b, o, p);
    return cudaGetLastError();
}

cudaError_t launch_walk(const void* in, const void* weights, conv_args p, cudaStream_t s) {
    using C = walk_cfg;
    static std::once_flag once;
    static cudaError_t attr = cudaSuccess;
    std::call_once(once, [] { attr = raise_smem(conv3x3_walk, C::SMEM); });
    if (attr != cudaSuccess) return attr;
    CUtensorMap a, b, o{};
    const cuuint64_t w2 = p.w / 2, rows_n = (cuuint64_t)p.n_img * p.h, pitch = (cuuint64_t)p.out_cstride * 2;
    p.tiles_x = (p.w / 2 + 127) / 128;
    {
        cuuint64_t dims[4] = {64, w2, (cuuint64_t)p.h, (cuuint64_t)p.n_img}, str[3] = {128, w2 * 128, (cuuint64_t)p.h * w2 * 128};
        cuuint32_t box[4] = {64, 136, 1, 1};
        cuuint64_t dw[2] = {9 * 32, (cuuint64_t)p.cout}, sw[1] = {9 * 32 * 2};
        cuuint32_t bw[2] = {32, 32};
        if (!make_map(&a, in, 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B) ||
            !make_map(&b, weights, 2, dw, sw, bw, CU_TENSOR_MAP_SWIZZLE_64B))
            return cudaErrorInvalidValue;
    }
    if (p.tma_out && p.out_cstride == 32) {
        cuuint64_t dims[3] = {64, w2, rows_n}, str[2] = {128, w2 * 128};
        cuuint32_t box[3] = {64, 128, 1};
        if (!make_map(&o, p.out, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return cudaErrorInvalidValue;
    } else if (p.tma_out) {
        // a channel slice: the left and the right pixels of the pairs
        cuuint64_t dims[5] = {(cuuint64_t)p.out_cstride, 2, w2, 1, rows_n};
        cuuint64_t str[4] = {pitch, 2 * pitch, 2 * w2 * pitch, 2 * w2 * pitch};
        cuuint32_t box[5] = {32, 1, 128, 1, 1};
        if (!make_map(&o, p.out, 5, dims, str, box, CU_TENSOR_MAP_SWIZZLE_64B)) return cudaErrorInvalidValue;
    }
    const int ntn = p.cout / 32, sms = sm_count_cached();
    // rows per band: the least rows of the busiest strip, each band's two halo rows
    // included; two strips per CTA, no band of one row
    const long long strips = (long long)p.n_img * p.tiles_x, ctas = std::max(1, sms / ntn);
    if (strips * p.h > 0x7FFFFFFFLL) return cudaErrorInvalidValue;
    long long best = -1;
    for (long long nb = 1; nb <= 16 * ctas / strips + 8 && nb <= (p.h + 1) / 2; nb++) {
        int band = (int)((p.h + nb - 1) / nb);
        if (p.pool) band = (band + 1) / 2 * 2;
        if (p.h % band == 1 || band < 2) continue;
        const long long tasks = strips * ((p.h + band - 1) / band), cost = (tasks + 2 * ctas - 1) / (2 * ctas) * (band + 2);
        if (best < 0 || cost < best) {
            best = cost;
            p.band = band;
        }
    }
    const long long tasks = strips * ((p.h + p.band - 1) / p.band);
    const int grid = (int)std::min<long long>(tasks, ctas) * ntn;
    conv3x3_walk<<<grid, 320, C::SMEM, s>>>(a, b, o, p);
    return cudaGetLastError();
}

int pick_bn(int c) {
    for (int bn : {256, 128, 64, 32})
        if (c % bn == 0) return bn;
    return 0;
}

template <int CO, int BN>
cudaError_t launch_wgrad_rows(const void* dy, const void* x, int x_cstride, wgrad_args p, cudaStream_t s) {
    using C = wgrad_rows_cfg<CO, BN>;
    static std::once_flag once;
    static cudaError_t attr = cudaSuccess;
    std::call_once(once, [] { attr = raise_smem(wgrad3x3_rows<CO, BN>, C::SMEM); });
    if (attr != cudaSuccess) return attr;
    CUtensorMap ma, mb;
    const CUtensorMapSwizzle swa = CO == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
    const CUtensorMapSwizzle swb = BN == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
    const cuuint64_t w = p.w, h = p.h, n = p.n_img, xp = (cuuint64_t)x_cstride * 2;
    cuuint64_t da[4] = {CO, w, h, n}, sa[3] = {CO * 2, w * CO * 2, h * w * CO * 2};
    cuuint64_t db[4] = {(cuuint64_t)x_cstride, w, h, n}, sb[3] = {xp, w * xp, h * w * xp};
    cuuint32_t ba[4] = {CO, 64, C::R + 2, 1}, bb[4] = {BN, 72, C::R, 1};
    if (!make_map(&ma, dy, 4, da, sa, ba, swa) || !make_map(&mb, x, 4, db, sb, bb, swb)) return cudaErrorInvalidValue;
    const long long total = (long long)p.n_img * ((p.h + C::R - 1) / C::R) * (p.w / 64);
    if (total > 0x7FFFFFFFLL) return cudaErrorInvalidValue;
    p.total = (int)total;
    // every SM full once (two CTAs: twice). The rounding error of a sum grows with its
    // length: 16 images of 256 x 256, 64 -> 64: 7.0e-6 relative, 8.0e-6 with a box and a
    // launch per tap.
    const int ntiles = p.cin / BN;
    const int splits = (int)std::min<long long>(total, std::max(1, sm_count_cached() * C::CTAS * (C::CTAS == 2 ? 2 : 1) / ntiles));
    p.kpc = (p.total + splits - 1) / splits;
    dim3 grid((unsigned)((p.total + p.kpc - 1) / p.kpc), (unsigned)ntiles);
    wgrad3x3_rows<CO, BN><<<grid, 128, C::SMEM, s>>>(ma, mb, p);
    return cudaGetLastError();
}

cudaError_t launch_wgrad_cols(const void* dy, const void* x, int x_cstride, wgrad_args p, cudaStream_t s) {
    using C = wgrad_cols_cfg;
    static std::once_flag once;
    static cudaError_t attr = cudaSuccess;
    std::call_once(once, [] { attr = raise_smem(wgrad3x3_cols, C::SMEM); });
    if (attr != cudaSuccess) return attr;
    CUtensorMap ma, mb;
    const cuuint64_t w = p.w, h = p.h, n = p.n_img, xp = (cuuint64_t)x_cstride * 2, yp = (cuuint64_t)p.cout * 2;
    cuuint64_t da[4] = {(cuuint64_t)p.cout, w, h, n}, sa[3] = {yp, w * yp, h * w * yp};
    cuuint64_t db[4] = {(cuuint64_t)x_cstride, w, h, n}, sb[3] = {xp, w * xp, h * w * xp};
    cuuint32_t ba[4] = {64, 64, 1, 1}, bb[4] = {32, 72, 1, 1};
    if (!make_map(&ma, dy, 4, da, sa, ba, CU_TENSOR_MAP_SWIZZLE_128B) || !make_map(&mb, x, 4, db, sb, bb, CU_TENSOR_MAP_SWIZZLE_64B))
        return cudaErrorInvalidValue;
    const long long total = (long long)p.n_img * p.h * (p.w / 64);
    if (total > 0x7FFFFFFFLL) return cudaErrorInvalidValue;
    p.total = (int)total;
    // Partial sums of at least two waves of CTAs: the rounding error of a sum grows
    // with its length (16 images of 128 x 128, 128 -> 128: 84.6 us and a relative error
    // of 5.8e-6 with one wave, 99.0 and 2.6e-6 with two, 111 and 1.7e-6 with three; 4.8e-6
    // with the boxes per tap). And at least the 45 for each 256 input channels that the
    // boxes per tap had, for at 256 -> 256 (64 x 64) two waves are fewer: 92.8 us and
    // 2.6e-6, with 45 103.1 and 1.7e-6, with 90 119.5 and 0.9e-6, the boxes 193 and 2.1e-6.
    const int mtiles = (p.cout + 127) / 128, tiles = mtiles * (p.cin / C::BN), sms = sm_count_cached();
    const int least = (45 + mtiles * (p.cin / pick_bn(p.cin)) - 1) / (mtiles * (p.cin / pick_bn(p.cin)));
    const int waves = std::max(2, (least * tiles + sms - 1) / sms);
    const int splits = (int)std::min<long long>(total, std::max(1, waves * sms / tiles));
    p.kpc = (p.total + splits - 1) / splits;
    dim3 grid((unsigned)((p.total + p.kpc - 1) / p.kpc), (unsigned)tiles);
    wgrad3x3_cols<<<grid, 128, C::SMEM, s>>>(ma, mb, p);
    return cudaGetLastError();
}

cudaError_t launch_wgrad(const void* dy, const void* x, int x_cstride, int x_coff, int n_img, int h, int w, int cout, int cin,
                         float* dw, float* db, double* db64, int* err, cudaStream_t s) {
    if (w % 64 || cin % 32 || cout <= 0 || cout % 32 || n_img <= 0 || h <= 0) return cudaErrorInvalidValue;
    if (x_coff % 32 || x_cstride % 32 || x_coff + cin > x_cstride) return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(x)) & 63) return cudaErrorMisalignedAddress;
    wgrad_args p{};
    p.n_img = n_img;
    p.h = h;
    p.w = w;
    p.cout = cout;
    p.cin = cin;
    p.x_coff = x_coff;
    p.dw = dw;
    p.db = db;
    p.db64 = db64;
    p.vec = (reinterpret_cast<uintptr_t>(dw) & 15) == 0;
    p.err = err;
    if (cout > 64) return launch_wgrad_cols(dy, x, x_cstride, p, s);
    if (cout == 32)
        return cin % 64 ? launch_wgrad_rows<32, 32>(dy, x, x_cstride, p, s) : launch_wgrad_rows<32, 64>(dy, x, x_cstride, p, s);
    return cin % 64 ? launch_wgrad_rows<64, 32>(dy, x, x_cstride, p, s) : launch_wgrad_rows<64, 64>(dy, x, x_cstride, p, s);
}

}  // namespace

extern "C" cudaError_t rfk_unet_conv3x3(const void* in, int n_img, int h, int w, int in_cstride, int in_coff, int cin,
                                        const void* weights, int cout, const float* bias, int flags, void* out,
                                        int out_cstride, int out_coff, const void* mask, int mask_cstride, int mask_coff,
                                        int accumulate, int* err, cudaStream_t s) {
    return rfk_unet_conv3x3_pool(in, n_img, h, w, in_cstride, in_coff, cin, weights, cout, bias, flags, out, out_cstride, out_coff,
                                 mask, mask_cstride, mask_coff, accumulate, nullptr, err, s);
}

extern "C" cudaError_t rfk_unet_conv3x3_pool(const void* in, int n_img, int h, int w, int in_cstride, int in_coff, int cin,
                                             const void* weights, int cout, const float* bias, int flags, void* out,
                                             int out_cstride, int out_coff, const void* mask, int mask_cstride, int mask_coff,
                                             int accumulate, void* pool, int* err, cudaStream_t s) {
    const bool rgb = (flags & RFK_UNET_RGBOUT) != 0;
    if (cin % 32 || in_coff % 32 || in_cstride % 32 || cout % 32) return cudaErrorInvalidValue;
    if (rgb ? accumulate || out_coff || out_cstride != 4 : out_coff % 32 || out_cstride % 32 || out_coff + cout > out_cstride)
        return cudaErrorInvalidValue;
    if (mask && (mask_coff % 32 || mask_cstride % 32)) return cudaErrorInvalidValue;
    if (in_coff + cin > in_cstride || n_img <= 0 || h <= 0 || w <= 0) return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(weights) | reinterpret_cast<uintptr_t>(out)) & 63)
        return cudaErrorMisalignedAddress;
    const bool wide_k = cin % 64 == 0 && in_coff % 64 == 0;
    // Order of the sums: an accumulator adds its products in one order, whichever
    // sizes and whichever kernel: channel block, tap (32 output channels), tap row,
    // channel block, column tap (64), or tap, channel block (128, 256). So an image
    // denoised is the image whose loss is computed, bit for bit, and losses are
    // reproducible. A row-streaming kernel that summed the tap rows in accumulators of
    // their own took a 1080p denoise from 1.09 to 0.97 ms and moved its half-float
    // channels by up to 0.007 (3e-4 relative over the image).
    const bool up2 = (flags & RFK_UNET_UP2) != 0;
    // 32 dense input channels: conv3x3_walk, if the tiles below would be of 32 output
    // channels (32 f32 channels out: slower than the tiles)
    const bool walk = !up2 && !accumulate && !(flags & RFK_UNET_F32OUT) && cin == 32 && in_cstride == 32 && w % 2 == 0 &&
                      h >= 2 && pick_bn(cout) == 32;
    if (pool && (!walk || h % 2)) return cudaErrorInvalidValue;
    const int bn = pick_bn(cout);
    // tap reuse: 32 output channels (4 rows per tile) load each input channel
    // block once for all nine taps (MODE 2, 32-channel K blocks so that three
    // 52 KB stages fit; it keeps one output tile's weights resident: cout == 32,
    // at most 3 input blocks); 64 (2 rows) once per tap row (MODE 1); 128 (2 rows
    // sharing each weight tile) once per tap row if there is one channel block, 256 (1
    // row) once per tap (MODE 0: three 32 KB weight tiles and the row leave one stage).
    const int mode2 = cout == 32 && cin <= 32 * 3;
    const int bk = !mode2 && wide_k ? 64 : 32;
    const int mode = mode2 ? 2 : bn <= 64 ? 1 : bn == 128 && cin == bk ? 1 : 0;
    CUtensorMap ma, mb;
    const CUtensorMapSwizzle sw = bk == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
    {
        cuuint64_t dims[4] = {(cuuint64_t)in_cstride, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n_img};
        cuuint64_t str[3] = {(cuuint64_t)in_cstride * 2, (cuuint64_t)w * in_cstride * 2, (cuuint64_t)h * w * in_cstride * 2};
        // image rows and pixel lines of an A box, as conv_cfg<BK, BN, MODE>
        const cuuint32_t box_rows = bn == 256 ? 1u : bn == 128 ? 2u : (cuuint32_t)(128 / bn) + (mode == 2 ? 2u : 0u);
        cuuint32_t box[4] = {(cuuint32_t)bk, mode ? 136u : 128u, box_rows, 1};
        if (!make_map(&ma, in, 4, dims, str, box, sw)) return cudaErrorInvalidValue;
    }
    {
        cuuint64_t dims[2] = {(cuuint64_t)9 * cin, (cuuint64_t)cout};
        cuuint64_t str[1] = {(cuuint64_t)9 * cin * 2};
        cuuint32_t box[2] = {(cuuint32_t)bk, (cuuint32_t)bn};
        if (!make_map(&mb, weights, 2, dims, str, box, sw)) return cudaErrorInvalidValue;
    }
    conv_args p{};
    p.n_img = n_img;
    p.h = h;
    p.w = w;
    p.tiles_x = (w + 127) / 128;
    p.cin = cin;
    p.cin_off = in_coff;
    p.cout = cout;
    p.out = out;
    p.out_cstride = out_cstride;
    p.out_coff = out_coff;
    p.bias = bias;
    p.relu = flags & RFK_UNET_RELU;
    p.out_rgb = rgb;
    p.out_f32 = rgb || (flags & RFK_UNET_F32OUT);
    p.up2 = up2;
    if (p.up2 && (p.out_f32 || accumulate)) return cudaErrorInvalidValue;
    p.mask = static_cast<const bf16*>(mask);
    p.mask_cstride = mask_cstride;
    p.mask_coff = mask_coff;
    p.accumulate = accumulate;
    p.err = err;
    p.tma_out = !p.out_f32 && !accumulate;
    p.pool = static_cast<bf16*>(pool);
    if (walk) return launch_walk(in, weights, p, s);
    CUtensorMap mo{};
    if (p.tma_out) {
        // output rows of all images one after another; with up2 as (channel, x
        // parity, x, y parity, y) of the (2h, 2w) image. Boxes of 128 pixels x 64 or
        // 32 channels, as conv_cfg::OC; pixels past the width are clipped.
        const cuuint32_t oc = bn % 64 == 0 ? 64u : 32u;
        const CUtensorMapSwizzle osw = oc == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
        const cuuint64_t pitch = (cuuint64_t)out_cstride * 2, rows_n = (cuuint64_t)n_img * h;
        bool good;
        if (p.up2) {
            cuuint64_t dims[5] = {(cuuint64_t)out_cstride, 2, (cuuint64_t)w, 2, rows_n};
            cuuint64_t str[4] = {pitch, 2 * pitch, 2 * (cuuint64_t)w * pitch, 4 * (cuuint64_t)w * pitch};
            cuuint32_t box[5] = {oc, 1, 128, 1, 1};
            good = make_map(&mo, out, 5, dims, str, box, osw);
        } else {
            cuuint64_t dims[3] = {(cuuint64_t)out_cstride, (cuuint64_t)w, rows_n};
            cuuint64_t str[2] = {pitch, (cuuint64_t)w * pitch};
            cuuint32_t box[3] = {oc, 128, 1};
            good = make_map(&mo, out, 3, dims, str, box, osw);
        }
        if (!good) return cudaErrorInvalidValue;
    }
    if (bk == 64) {
        switch (bn) {
        case 256: return launch_conv<64, 256, 0>(ma, mb, mo, p, s);
        case 128: return mode ? launch_conv<64, 128, 1>(ma, mb, mo, p, s) : launch_conv<64, 128, 0>(ma, mb, mo, p, s);
        case 64: return launch_conv<64, 64, 1>(ma, mb, mo, p, s);
        default: return launch_conv<64, 32, 1>(ma, mb, mo, p, s);
        }
    }
    switch (bn) {
    case 256: return launch_conv<32, 256, 0>(ma, mb, mo, p, s);
    case 128: return mode ? launch_conv<32, 128, 1>(ma, mb, mo, p, s) : launch_conv<32, 128, 0>(ma, mb, mo, p, s);
    case 64: return launch_conv<32, 64, 1>(ma, mb, mo, p, s);
    default: return mode == 2 ? launch_conv<32, 32, 2>(ma, mb, mo, p, s) : launch_conv<32, 32, 1>(ma, mb, mo, p, s);
    }
}

extern "C" cudaError_t rfk_unet_wgrad3x3(const void* dy, const void* x, int x_cstride, int x_coff, int n_img, int h, int w,
                                         int cout, int cin, float* dw, int* err, cudaStream_t s) {
    return launch_wgrad(dy, x, x_cstride, x_coff, n_img, h, w, cout, cin, dw, nullptr, nullptr, err, s);
}

extern "C" cudaError_t rfk_unet_wgrad3x3_bias(const void* dy, const void* x, int x_cstride, int x_coff, int n_img, int h, int w,
                                              int cout, int cin, float* dw, float* db, int* err, cudaStream_t s) {
    return launch_wgrad(dy, x, x_cstride, x_coff, n_img, h, w, cout, cin, dw, db, nullptr, err, s);
}

extern "C" cudaError_t rfk_unet_wgrad3x3_bias64(const void* dy, const void* x, int x_cstride, int x_coff, int n_img, int h, int w,
                                                int cout, int cin, float* dw, double* db, int* err, cudaStream_t s) {
    return launch_wgrad(dy, x, x_cstride, x_coff, n_img, h, w, cout, cin, dw, nullptr, db, err, s);
}
