// Inline-PTX wrappers for the Blackwell (sm_100 family) tensor-core path of the
// denoiser: mbarriers, TMA tiled loads, TMEM allocation, tcgen05.mma / commit /
// ld, and the shared-memory and instruction descriptors of tcgen05.mma.
//
// Descriptor layouts (PTX ISA, tcgen05 "shared memory descriptor" and
// "instruction descriptor" for .kind::f16):
//   smem descriptor (64 bit): [0,14) start address >> 4, [16,30) leading byte
//     offset >> 4, [32,46) stride byte offset >> 4, [46,48) version = 1,
//     [49,52) base offset, [52] LBO mode, [61,64) layout: 0 none,
//     2 128-byte swizzle, 4 64-byte swizzle, 6 32-byte swizzle.
//   instruction descriptor (32 bit): [4,6) D type (1 = f32), [7,10) A type
//     (1 = bf16), [10,13) B type, [15] A major (0 = K), [16] B major,
//     [17,23) N >> 3, [24,29) M >> 4.
// Every wait here is bounded: it gives up after kWaitNs of %globaltimer time
// (or kWaitIters polls) and reports failure, so that a kernel whose pipeline
// broke ends with an error status instead of hanging the GPU.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace tc {

constexpr unsigned long long kWaitNs = 2000000000ull;  // 2 s
constexpr uint32_t kWaitIters = 1u << 28;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait for the phase with the given parity; false after the limit.
// The usual wait ends within a few polls; %globaltimer is read only after 64 of
// them, for reading it takes longer than such a wait.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    for (int i = 0; i < 64; i++)
        if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = now_ns();
    for (uint32_t i = 1; i < kWaitIters; i++) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 63u) == 0 && now_ns() - t0 > kWaitNs) return false;
    }
    return false;
}

// TMA tiled loads into shared memory, completing on `bar` (complete_tx).
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"((uint64_t)map), "r"(c0), "r"(c1), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(smem_u32(dst)),
        "l"((uint64_t)map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
        : "memory");
}

// TMA tiled stores from shared memory (bulk groups of the issuing thread). The
// writes of other threads to the tile need fence_async() and a barrier first.
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, const void* src, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"((uint64_t)map),
                 "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}

__device__ __forceinline__ void tma_store_5d(const CUtensorMap* map, const void* src, int c0, int c1, int c2, int c3, int c4) {
    asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5, %6}], [%1];" ::"l"(
                     (uint64_t)map),
                 "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
                 : "memory");
}

__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// At most N of this thread's bulk groups still read shared memory / are unfinished.
template <int N>
__device__ __forceinline__ void tma_store_wait_read() {
    asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ void tma_store_wait() {
    asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// Barrier `id` (1-15) among `threads` threads of the block, whole warps. The
// warp is brought together before and after it: lanes come here from polling
// loops and single-lane branches, and what follows are .aligned instructions.
__device__ __forceinline__ void named_barrier(int id, int threads) {
    __syncwarp();
    asm volatile("barrier.cta.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
    __syncwarp();
}

// As named_barrier; whether `ok` holds in all of its threads.
__device__ __forceinline__ bool named_barrier_all(int id, int threads, bool ok) {
    uint32_t r;
    __syncwarp();
    asm volatile("{\n .reg .pred p, q;\n setp.ne.b32 p, %3, 0;\n barrier.cta.red.and.pred q, %1, %2, p;\n selp.u32 %0, 1, 0, q;\n}"
                 : "=r"(r)
                 : "r"(id), "r"(threads), "r"((uint32_t)ok)
                 : "memory");
    __syncwarp();
    return r != 0;
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// One full warp: allocate ncols TMEM columns (power of 2, >= 32); the base
// address goes to *dst in shared memory.
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// tcgen05.mma and commit take their operands from uniform registers. In a branch
// that one lane takes, the compiler keeps descriptors in per-lane registers and
// moves them over before every instruction, which made an MMA of 45-56 cycles
// take 120-160 to issue. So a whole warp runs the issuing loop, with warp-uniform
// operands and control flow (waits through all_lanes), and the instruction
// itself is predicated: `one` is nonzero in the issuing lane only.
// The descriptors' high words are constants of the layout and only the low words
// (start address, leading offset) are passed, for the same reason.
// D[tmem] (+)= A[smem] * B[smem]^T, bf16 inputs, f32 accumulator.
template <uint32_t AHI, uint32_t BHI>
__device__ __forceinline__ void mma_bf16(uint32_t one, uint32_t d_tmem, uint32_t alo, uint32_t blo, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p, q;\n .reg .b64 da, db;\n mov.b64 da, {%1, %6};\n mov.b64 db, {%2, %7};\n"
        " setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
        " @q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n}\n" ::"r"(d_tmem),
        "r"(alo), "r"(blo), "r"(idesc), "r"(accumulate), "r"(one), "n"(AHI), "n"(BHI)
        : "memory");
}

// Arrives on `bar` once every tcgen05.mma issued so far by the issuing lane is done.
__device__ __forceinline__ void mma_commit(uint32_t one, uint64_t* bar) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n"
        " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(smem_u32(bar)),
        "r"(one)
        : "memory");
}

// A wait of every lane of the warp; the same answer in all of them.
__device__ __forceinline__ bool all_lanes(bool ok) { return __all_sync(0xffffffffu, ok) != 0; }

// 32 consecutive f32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    __syncwarp();
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,"
        "%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

// Clears 32 consecutive columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_zero32(uint32_t taddr) {
    __syncwarp();
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,"
        "%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
        "r"(0u)
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// 16 consecutive f32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    __syncwarp();
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// Descriptor of an operand tile in shared memory that TMA wrote with a row of
// `row_bytes` (128 or 64) and the matching swizzle, as two words: the high word
// depends on the layout only, the low word on the start address.
// K-major: rows are `row_bytes` apart, 8-row groups (the swizzle atom)
// 8 * row_bytes apart (the stride byte offset; the leading one is unused).
// MN-major (the M or N index contiguous; boxes of row_bytes x K rows, one per
// group of row_bytes / 2 M or N elements, `group_stride` bytes apart): the
// stride byte offset is the 8-row K group, the leading byte offset the group
// stride (checked on the GPU against a reference product for both swizzles and
// one to four groups; a group stride of one row makes the groups the same rows
// from one pixel line later each, as the weight gradients' column taps).
// A start address may lie inside a tile that was written from a 1024-byte
// aligned base: whole rows (pixel lines) past it, plus 32-byte K steps within a
// row. The swizzle pattern is taken from the address bits of each access, as TMA
// applied it, so the matrix base offset field stays 0.
__host__ __device__ constexpr uint32_t desc_hi(uint32_t row_bytes) {
    return ((8u * row_bytes) >> 4) | (1u << 14) | ((row_bytes == 128 ? 2u : 4u) << 29);
}
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) { return ((saddr >> 4) & 0x3FFFu) | (1u << 16); }
__device__ __forceinline__ uint32_t desc_lo_mn(uint32_t saddr, uint32_t group_stride) {
    return ((saddr >> 4) & 0x3FFFu) | (((group_stride >> 4) & 0x3FFFu) << 16);
}

// bf16 x bf16 -> f32, both operands K-major, M x N tile.
__host__ __device__ constexpr uint32_t idesc_bf16(uint32_t m, uint32_t n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

// As idesc_bf16 with the B operand MN-major (bit 16).
__host__ __device__ constexpr uint32_t idesc_bf16_bmn(uint32_t m, uint32_t n) { return idesc_bf16(m, n) | (1u << 16); }

}  // namespace tc
