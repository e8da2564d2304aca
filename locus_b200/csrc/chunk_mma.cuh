// Portions of a recurrence in chunks of 16 tokens (gla.cu): small float32 matrix products on the tensor cores.
//
// Every float32 operand is cut into three bfloat16 whose sum it is (bf16_parts.cuh), and a product of two is the sum of six products
// of parts, the small ones first: it lacks at most 2^-24 of itself, and float32 sums round as ever.  mma.sync m16n8k16 (a warp's 16 x 16 times 16 x 8): lane 4 g + t holds of A the rows g and g + 8 at columns 2 t,
// 2 t + 1, 2 t + 8, 2 t + 9, of B the column g at the same rows, of the sums rows g and g + 8 at columns 2 t, 2 t + 1, so that the
// sums of two neighbouring tiles of eight columns are the A operand of a product over those sixteen columns.
#pragma once
#include "bf16_parts.cuh"
#include "walk.cuh"

#define CH 16   // tokens of a chunk

__device__ __forceinline__ void ch_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The parts of A and B of a product's six, from the smallest on.  Callers go through them for all their sums in turn: six MMAs
// on one sum wait for each other.  b: [part][k's lower and upper half]
template <int P>
__device__ __forceinline__ void ch_mma_part(float (&c)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][2]) {
    constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};
    ch_mma(c, a[PA[P]], b[PB[P]][0], b[PB[P]][1]);
}
// Two sums c[n] += A B[n].
__device__ __forceinline__ void ch_mma_pair(float (&c)[2][4], const uint32_t (&a)[3][4], const uint32_t (&b)[2][3][2]) {
#define CH_STEP(P) ch_mma_part<P>(c[0], a, b[0]); ch_mma_part<P>(c[1], a, b[1]);
    CH_STEP(0) CH_STEP(1) CH_STEP(2) CH_STEP(3) CH_STEP(4) CH_STEP(5)
#undef CH_STEP
}
// Four 8 x 8 tiles of bfloat16 from shared memory, lane l giving the address of row l & 7 of tile l >> 3; plain or transposed.
__device__ __forceinline__ uint32_t ch_smem(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void ch_ldsm(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(ch_smem(p)) : "memory");
}
__device__ __forceinline__ void ch_ldsm_t(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(ch_smem(p)) : "memory");
}
// Bulk copies into shared memory, counted by an mbarrier, and a bounded wait for them (about a second of clock cycles): when it runs out
// the module's error word is set, all later waits that have to spin return soon, and the caller goes on with what is there, so that the
// kernel ends.
#define CH_WAIT_LIMIT 2000000000LL
__device__ int g_chunk_error = 0;
__device__ __forceinline__ void ch_bar_init(uint32_t bar) { asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar)); }
__device__ __forceinline__ void ch_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
                 "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void ch_wait(uint32_t bar, uint32_t parity) {
    auto there = [&]() -> bool {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        return ok != 0;
    };
    if (there()) return;
    const long long t0 = clock64();
    for (int i = 1; !there(); ++i) {
        if ((i & 63) == 0 && *reinterpret_cast<volatile int*>(&g_chunk_error) != 0) return;   // (a trip to L2)
        if (clock64() - t0 > CH_WAIT_LIMIT) {
            atomicCAS(&g_chunk_error, 0, 1);
            return;
        }
    }
}
