// float32 products on the Blackwell tensor cores (included by gemm_simt.cu, whose arguments and epilogue it shares): every
// float32 is cut into three bfloat16 whose sum it is (bf16_parts.cuh, with the bound of what the six products of parts leave out of a
// product and the range that this holds for).  Products of bfloat16 are exact in the tensor cores; what rounds is their sum: a
// float32 accumulator is cut off, not rounded, at every 16 columns of k.  So the large products a0 b0 have an accumulator of their own,
// which is taken out after 64 columns and added up in registers, rounded; the five small ones share another one for
// the whole sum, where a cut is 2^-8 of what it would be beside the large ones.
//
//   D[n, t] (tensor memory: lane n, column t) = sum_k W[n0 + n, k] x[t0 + t, k]:  weights are the M side, tokens the N side
//
// A first kernel cuts the rows of x up (and gathers them), once for all weight rows.  Of the second's warps, 0 has the TMA fetch a
// stage, 32 columns of k: 128 weight rows as float32 and the three parts of the rows of x, swizzled (the B operand); 4 to 11 cut the
// weights up, a thread a row, into tensor memory (the A operand: read from there six times it takes none of the shared memory's
// bandwidth, which the operands of six products would exceed); 1 issues the MMAs; 12 to 15 take the accumulators
// out, add them up and do the epilogue while the next tile's MMAs run.  A SwiGLU tile holds 64 weight rows of each
// matrix.  A block walks over tiles, all roles run ahead across them.
//
// An operand that is not finite makes NaN of every sum it enters, and the rounded first parts of two values may be more than float32
// holds where their product is not (within 2^-7 of its largest value): a sum that is not finite is formed again, by plain
// multiply-adds, from its row and weight row, and comes out as such operands give it.
//
// What bounds it: the MMAs, six for one (a stage of 128 rows 768 cycles), where there are many rows, and the weights' way from
// memory where there are few.  Measured, against the CUDA-core kernel: 2,048 x 6,144 x 2,048 1,156 -> 246 us (209 TFLOP/s; cuBLAS's
// bfloat16 rate / 6 is 276), 512 x 6,144 x 2,048 301 -> 83, 64 x 6,144 x 2,048 47 -> 22, 512 x 2,048 x 5,632 268 -> 67, the routed
// experts of 512 tokens (60 x (2,048 -> 1,408 -> 2,048), 4 picks) 1,004 -> 445 (their weights 4.7 TB/s).  The error of
// sums of 2,048 normally distributed products against 64 bits 5.7e-7 -> 1.3e-7 of their norm (uncut; CUDA cores cut in parts
// 3.3e-7), of 128 1.5e-7 -> 0.75e-7; of one sign 3.5e-7 -> 1.2e-7 and 0.93e-7 -> 0.92e-7, where the CUDA cores' sums are short, though (512
// in 8 parts, 5,632 in 8), 0.56e-7 -> 0.90e-7 and 0.80e-7 -> 0.90e-7: what the accumulators cut off within 64 columns is of one sign then.
// With the large products' accumulator taken out after 128 columns 1.9e-7 and 1.25e-7 (the first two, first parts cut off), 3 % quicker.  On the way here: weights and x cut up
// by the same eight warps 573 us for the first (a chain of waits, loads, conversions and stores for every stage), x cut up
// first and the sums taken out by the same warps 321.
//
// Every wait on an mbarrier is bounded; when one runs out the module's error word is set, all later waits return at once and
// the kernel ends.
#pragma once
#include <cuda.h>
#include <string.h>

#include "bf16_parts.cuh"

#define FT_W 128              // weight rows of a tile
#define FT_K 32               // columns of k of a stage: 128 bytes of float32, 64 of bfloat16
#define FT_W_BYTES (FT_W * FT_K * 4)
#define FT_CHUNK 2            // stages whose large products share an accumulator
#define FT_THREADS 512        // four groups of four warps: load and MMA; two that cut weights up; sums and epilogue
#define FT_SUM 128            // threads that take accumulators out
#define FT_WAIT_LIMIT 2000000000LL

__device__ int g_f32_tc_error = 0;

__device__ __forceinline__ uint32_t ft_smem(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void ft_bar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void ft_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool ft_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait; false when the limit ran out here or anywhere else in the grid before.
__device__ __forceinline__ bool ft_wait(uint32_t bar, uint32_t parity, int code) {
    if (ft_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (int i = 1; !ft_try_wait(bar, parity); ++i) {
        if ((i & 63) == 0 && *reinterpret_cast<volatile int*>(&g_f32_tc_error) != 0) return false;   // (a trip to L2)
        if (clock64() - t0 > FT_WAIT_LIMIT) {
            atomicCAS(&g_f32_tc_error, 0, code);
            return false;
        }
    }
    return true;
}
// B operand: K-major rows of 64 bytes, 64-byte swizzle (16-byte piece c of row r lies at place c ^ (r / 2 & 3)), groups
// of 8 rows 512 bytes apart.
__device__ __forceinline__ uint64_t ft_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((saddr & 0x3FFFF) >> 4);
    d |= static_cast<uint64_t>(1) << 16;
    d |= static_cast<uint64_t>(512 >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(4) << 61;
    return d;
}
// D += A B, A in tensor memory
__device__ __forceinline__ void ft_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void ft_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void ft_ld32(uint32_t taddr, uint32_t* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,"
        "%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
}
__device__ __forceinline__ void ft_ld16(uint32_t taddr, uint32_t* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
}
__device__ __forceinline__ void ft_st8(uint32_t taddr, const uint32_t* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ bool ft_odd(float v) { return !(fabsf(v) < INFINITY); }
// A sum that came out as not finite, formed by multiply-adds.
__device__ __forceinline__ float ft_plain(const float* x, const float* w, int n) {
    float even = 0.f, odd = 0.f;
#pragma unroll 1
    for (int k = 0; k < n; k += 2) {   // n is a multiple of 4
        even = fmaf(x[k], w[k], even);
        odd = fmaf(x[k + 1], w[k + 1], odd);
    }
    return even + odd;
}

struct FtGeom {
    int row0, rows, n0, w_off, kb0, n_kb, split;   // rows of x, first output column, first weight row of the expert, stages
};

// The three parts of x, [part][row][Kp] with Kp = K rounded up to whole stages (zeros behind K): a thread cuts eight columns.
__global__ void __launch_bounds__(256) f32_cut_kernel(const float* __restrict__ x, long long ldx, const int* __restrict__ x_rows,
                                                      int x_row_div, int K, int Kp, int rows, bf16* __restrict__ parts) {
    const long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
    const int per = Kp / 8, row = static_cast<int>(i / per), k = static_cast<int>(i - static_cast<long long>(row) * per) * 8;
    if (row >= rows) return;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4* p = reinterpret_cast<const float4*>(x + (x_rows ? x_rows[row] / x_row_div : row) * ldx + k);
    const float4 u = k < K ? p[0] : z, v = k + 4 < K ? p[1] : z;
    uint4 q[3];
    bf16_parts(u.x, u.y, q[0].x, q[1].x, q[2].x);
    bf16_parts(u.z, u.w, q[0].y, q[1].y, q[2].y);
    bf16_parts(v.x, v.y, q[0].z, q[1].z, q[2].z);
    bf16_parts(v.z, v.w, q[0].w, q[1].w, q[2].w);
#pragma unroll
    for (int j = 0; j < 3; ++j) *reinterpret_cast<uint4*>(parts + (static_cast<long long>(j) * rows + row) * Kp + k) = q[j];
}

// TN: rows of x of a tile (64 or 128).
template <int TN>
struct FtShape {
    static constexpr int SA = TN == 128 ? 2 : 4;             // stages of cut weights (tensor memory)
    static constexpr int XB = TN * FT_K * 2;                 // bytes of a part of x
    static constexpr int STAGE = FT_W_BYTES + 3 * XB;
    static constexpr int SR = TN == 128 ? 4 : 6;             // stages of operands (shared memory)
    static constexpr int BARS = 8 * (2 * SR + SA + 5) + 8;
    static constexpr int SMEM = 1024 + SR * STAGE + 64 * FT_W * 4 + BARS;
};
// Boxes of a quarter, half, three quarters and all of a tile's rows of x.
struct FtXMaps {
    CUtensorMap m[4];
};

template <int TN, bool SWIGLU>
__global__ void __launch_bounds__(FT_THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_w2,
                   const __grid_constant__ FtXMaps maps_x, GemmArgs a, int tiles_x, int tiles_y) {
    using S = FtShape<TN>;
    constexpr int SA = S::SA, SR = S::SR, COLS = SWIGLU ? FT_W / 2 : FT_W;
    constexpr int T_CORR = 2 * TN, T_A = 3 * TN;   // tensor memory: large sums (two buffers), small sums, the weights' parts
    static_assert(T_A + SA * 48 <= 512, "tensor memory");
    extern __shared__ __align__(1024) uint8_t ft_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t raw = ft_smem(ft_raw), base = (raw + 1023u) & ~1023u;
    const uint32_t sSum = base + SR * S::STAGE, bars = sSum + 64 * FT_W * 4;   // a stage: weights, then x
    const uint32_t full = bars, free_ = full + 8 * SR, a_full = free_ + 8 * SR;
    const uint32_t m_full = a_full + 8 * SA, m_free = m_full + 16, c_free = m_free + 16, slot = c_free + 8;
    uint8_t* smem = ft_raw + (base - raw);

    if (threadIdx.x == 0) {
        for (int s = 0; s < SR; ++s) {
            ft_bar_init(full + 8 * s, 1);
            ft_bar_init(free_ + 8 * s, 1);    // a stage's MMAs are finished: its place in the ring and its parts' in tensor memory
        }
        for (int s = 0; s < SA; ++s) ft_bar_init(a_full + 8 * s, 4);
        for (int s = 0; s < 2; ++s) {
            ft_bar_init(m_full + 8 * s, 1);
            ft_bar_init(m_free + 8 * s, FT_SUM / 32);
        }
        ft_bar_init(c_free, FT_SUM / 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + (slot - base));

    const bool grouped = a.tile_expert != nullptr;
    const int n_y = grouped ? min(tiles_y, *a.n_tiles) : tiles_y;
    const int n_total = tiles_x * n_y * a.splits;   // the host refuses 2^31 or more
    const int n_all = (a.K + FT_K - 1) / FT_K, per_split = (n_all + a.splits - 1) / a.splits;
    auto stages_of = [&](int t) -> int { return max(0, min(per_split, n_all - t % a.splits * per_split)); };
    // Tiles that share weights run together: the row tiles of a plain product vary fastest; an expert's (it seldom has two)
    // follow each other.
    auto geom = [&](int t) -> FtGeom {
        FtGeom g;
        g.n_kb = stages_of(t);
        g.split = t % a.splits;
        g.kb0 = g.split * per_split;
        t /= a.splits;
        int tx, ty;
        if (grouped) {
            ty = t / tiles_x;
            tx = t - ty * tiles_x;
            g.row0 = a.tile_row0[ty];
            g.rows = a.tile_rows[ty];
            g.w_off = a.tile_expert[ty] * a.N;   // the host refuses weights of 2^31 rows or more
        } else {
            tx = t / tiles_y;
            ty = t - tx * tiles_y;
            g.row0 = ty * TN;
            g.rows = min(TN, a.M - g.row0);
            g.w_off = 0;
        }
        g.n0 = tx * COLS;
        return g;
    };

    // Registers by role: of the 128 a thread that the block was launched with, what the other groups give back goes to the sums
    // (64 + 2 x 104 + 232 <= 4 x 128).
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
        if (warp == 0 && lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < n_total && ok; t += gridDim.x) {
                const FtGeom g = geom(t);
                const int quarters = (g.rows + TN / 4 - 1) / (TN / 4);   // 1 .. 4
                const CUtensorMap* map_x = &maps_x.m[quarters - 1];
                const uint32_t bytes = FT_W_BYTES + quarters * (3 * S::XB / 4);
                for (int kb = g.kb0; kb < g.kb0 + g.n_kb; ++kb, ++it) {
                    const uint32_t s = it % SR, bar = full + 8 * s, dst = base + s * S::STAGE;
                    if (!ft_wait(free_ + 8 * s, ((it / SR) & 1) ^ 1, 1)) {
                        ok = false;
                        break;
                    }
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
                    auto load_w = [&](uint32_t to, const CUtensorMap* map) {
                        asm volatile(
                            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                            ::"r"(to), "l"(map), "r"(kb * FT_K), "r"(g.w_off + g.n0), "r"(bar)
                            : "memory");
                    };
                    load_w(dst, &map_w);
                    if (SWIGLU) load_w(dst + FT_W_BYTES / 2, &map_w2);
                    asm volatile(
                        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                        ::"r"(dst + FT_W_BYTES), "l"(map_x), "r"(kb * FT_K), "r"(g.row0), "r"(0), "r"(bar)
                        : "memory");
                }
            }
        } else if (warp == 1) {
            // (The whole warp walks, one thread issues: what does not depend on the lane stays in uniform registers.)
            uint32_t it = 0, chunk = 0, tiles = 0, elected;
            asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
            const uint64_t desc0 = ft_desc(base + FT_W_BYTES);
            for (int t = blockIdx.x; t < n_total; t += gridDim.x) {
                const FtGeom g = geom(t);
                if (g.n_kb == 0) continue;   // a part without a column
                // N covers the tile's live rows, in sixteens
                const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>((g.rows + 15) >> 4) << 18) |
                                       (static_cast<uint32_t>(FT_W >> 4) << 24);
                const uint32_t part = (static_cast<uint32_t>(g.rows + TN / 4 - 1) / (TN / 4)) * (S::XB / 4) >> 4;   // (of a box)
                ft_wait(c_free, (tiles & 1) ^ 1, 2);
                ++tiles;
                for (int kb = 0; kb < g.n_kb; ++kb, ++it) {
                    const bool first = kb % FT_CHUNK == 0, last = kb % FT_CHUNK == FT_CHUNK - 1 || kb == g.n_kb - 1;
                    const uint32_t s = it % SA, r = it % SR, buf = chunk & 1;
                    if (first) ft_wait(m_free + 8 * buf, ((chunk >> 1) & 1) ^ 1, 3);
                    ft_wait(a_full + 8 * s, (it / SA) & 1, 4);   // (the weights came with x)
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t tM = tmem + buf * TN, tC = tmem + T_CORR, tA = tmem + T_A + s * 48;
                    const uint64_t bx = desc0 + r * (S::STAGE >> 4);
                    if (elected) {
#pragma unroll
                        for (int ks = 0; ks < 2; ++ks) {
                            const uint32_t a0 = tA + 8 * ks, a1 = a0 + 16, a2 = a0 + 32;
                            const uint64_t b0 = bx + 2 * ks, b1 = b0 + part, b2 = b1 + part;
                            ft_mma(tC, a0, b2, idesc, kb > 0 || ks > 0);
                            ft_mma(tC, a2, b0, idesc, 1);
                            ft_mma(tC, a1, b1, idesc, 1);
                            ft_mma(tC, a0, b1, idesc, 1);
                            ft_mma(tC, a1, b0, idesc, 1);
                            ft_mma(tM, a0, b0, idesc, !first || ks > 0);
                        }
                        ft_commit(free_ + 8 * r);
                        if (last) ft_commit(m_full + 8 * buf);
                    }
                    __syncwarp();
                    if (last) ++chunk;
                }
            }
        }
    } else if (warp < 12) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 104;");
        // The first four of these warps take a tile's even stages, the others the odd ones, so that one group's chain of waits,
        // loads and stores runs beside the other's.
        const int quarter = warp & 3, wrow = quarter * 32 + lane;   // this thread's weight row
        const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
        uint32_t it = 0;
        for (int t = blockIdx.x; t < n_total; t += gridDim.x) {
            const int n_kb = stages_of(t);
            for (int kb = (warp >> 2) - 1; kb < n_kb; kb += 2) {
                const uint32_t i0 = it + kb, s = i0 % SA, r = i0 % SR;
                ft_wait(full + 8 * r, (i0 / SR) & 1, 7);
                const uint8_t* wr = smem + r * S::STAGE + wrow * 128;
                uint32_t p[2][3][8];   // the three parts of twice sixteen columns (what an MMA takes)
#pragma unroll
                for (int half = 0; half < 2; ++half)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float4 wv = *reinterpret_cast<const float4*>(wr + (((4 * half + i) ^ (wrow & 7)) << 4));
                        bf16_parts(wv.x, wv.y, p[half][0][2 * i], p[half][1][2 * i], p[half][2][2 * i]);
                        bf16_parts(wv.z, wv.w, p[half][0][2 * i + 1], p[half][1][2 * i + 1], p[half][2][2 * i + 1]);
                    }
                if (i0 >= SA) ft_wait(free_ + 8 * ((i0 - SA) % SR), ((i0 - SA) / SR) & 1, 6);   // the place of the stage SA before
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t tA = tmem + lanes + T_A + s * 48;
#pragma unroll
                for (int half = 0; half < 2; ++half)
#pragma unroll
                    for (int j = 0; j < 3; ++j) ft_st8(tA + 8 * half + 16 * j, p[half][j]);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) ft_arrive(a_full + 8 * s);
            }
            it += n_kb;
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
        const int quarter = warp & 3, tid = quarter * 32 + lane;   // this thread's weight row
        const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
        const float* X = static_cast<const float*>(a.x);
        float* sums = reinterpret_cast<float*>(smem + (sSum - base));   // [64][128]
        uint32_t m_done = 0;
        for (int t = blockIdx.x; t < n_total; t += gridDim.x) {
            const FtGeom g = geom(t);
            float acc[TN];
#pragma unroll
            for (int i = 0; i < TN; ++i) acc[i] = 0.f;
            auto add_up = [&](uint32_t from) {
#pragma unroll
                for (int c = 0; c < TN; c += 32) {
                    if (c >= g.rows) break;   // (uniform: no live rows there)
                    uint32_t v[32];
                    ft_ld32(tmem + lanes + from + c, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 32; ++i) acc[c + i] += __uint_as_float(v[i]);
                }
            };
            const int chunks = (g.n_kb + FT_CHUNK - 1) / FT_CHUNK;
            for (int j = 0; j < chunks; ++j, ++m_done) {
                const uint32_t buf = m_done & 1;
                ft_wait(m_full + 8 * buf, (m_done >> 1) & 1, 5);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                add_up(buf * TN);
                if (j == chunks - 1) add_up(T_CORR);
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    ft_arrive(m_free + 8 * buf);
                    if (j == chunks - 1) ft_arrive(c_free);
                }
            }
            // The epilogue: 64 rows at a time through shared memory to a loop over eight of a column, whose arithmetic is independent.
            const int c = tid % COLS, n = g.n0 + c;
            const bool whole = SWIGLU || a.part == nullptr;
            const float b = n < a.N ? bias_of(a, n) : 0.f, b2 = a.act == 4 && n < a.N ? bias_of(a, a.N + n) : 0.f;
            const int k0 = g.kb0 * FT_K, kn = min(a.K, (g.kb0 + g.n_kb) * FT_K) - k0;
#pragma unroll
            for (int pass = 0; pass < TN / 64; ++pass) {
                if (pass * 64 >= g.rows) break;
                if (SWIGLU) asm volatile("bar.sync 1, %0;" ::"n"(FT_SUM) : "memory");   // the rows before are read
#pragma unroll
                for (int i = 0; i < 64; ++i) sums[i * FT_W + tid] = acc[64 * pass + i];
                if (SWIGLU) asm volatile("bar.sync 1, %0;" ::"n"(FT_SUM) : "memory");   // (else a thread reads what it wrote)
                const int m_end = min(64, g.rows - 64 * pass), row0 = g.row0 + 64 * pass;
                if (n < a.N)
#pragma unroll 1
                    for (int m0 = 8 * (tid / COLS); m0 < m_end; m0 += 8 * (FT_SUM / COLS)) {
                        const int live = min(8, m_end - m0);
                        float v[8], v2[8];
                        bool odd = false;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            v[i] = sums[(m0 + i) * FT_W + c];
                            if (SWIGLU) v2[i] = sums[(m0 + i) * FT_W + COLS + c];
                            odd |= ft_odd(v[i]) || (SWIGLU && ft_odd(v2[i]));
                        }
                        if (odd)
#pragma unroll 1
                            for (int q = 0; q < live; ++q) {
                                const int r = row0 + m0 + q;
                                const float* xp = X + static_cast<long long>(a.x_rows ? a.x_rows[r] / a.x_row_div : r) * a.ldx + k0;
                                const long long wo = static_cast<long long>(g.w_off + n) * a.K + k0;
                                const float s1 = ft_plain(xp, static_cast<const float*>(a.w) + wo, kn);
                                const float s2 = SWIGLU ? ft_plain(xp, static_cast<const float*>(a.w2) + wo, kn) : 0.f;
#pragma unroll
                                for (int i = 0; i < 8; ++i)   // (the array stays in registers)
                                    if (i == q && (ft_odd(v[i]) || (SWIGLU && ft_odd(v2[i])))) {
                                        v[i] = s1;
                                        if (SWIGLU) v2[i] = s2;
                                    }
                            }
                        if (!whole) {
                            float* to = a.part + (static_cast<size_t>(g.split) * a.M + row0 + m0) * a.N + n;
#pragma unroll
                            for (int i = 0; i < 8; ++i, to += a.N)
                                if (i < live) *to = v[i];
                            continue;
                        }
                        float rs[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) rs[i] = 1.f;
                        if (a.row_scale)
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                if (i < live) rs[i] = scale_of(a, row0 + m0 + i);
                        if (a.act == 0) {
#pragma unroll
                            for (int i = 0; i < 8; ++i) v[i] = ((SWIGLU ? v[i] / (1.0f + expf(-v[i])) * v2[i] : v[i]) + b) * rs[i];
                        } else {
#pragma unroll
                            for (int i = 0; i < 8; ++i) v[i] = finish<SWIGLU>(a, rs[i], v[i], SWIGLU ? v2[i] : 0.f, b, b2);
                        }
                        const size_t o = static_cast<size_t>(row0 + m0) * a.ldo + n;
                        if (a.accumulate) {
                            float* to = static_cast<float*>(a.out) + o;
                            float old[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                if (i < live) old[i] = to[i * a.ldo];
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                if (i < live) to[i * a.ldo] = old[i] + v[i];
                        } else if (a.out_dt == LOCUS_DT_F32) {
                            float* to = static_cast<float*>(a.out) + o;
#pragma unroll
                            for (int i = 0; i < 8; ++i, to += a.ldo)
                                if (i < live) *to = v[i];
                        } else {
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                if (i < live) static_cast<bf16*>(a.out)[o + i * a.ldo] = __float2bfloat16_rn(v[i]);
                        }
                    }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

typedef CUresult (*FtEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static FtEncodeFn ft_encode_fn() {
    static FtEncodeFn fn = nullptr;
    if (fn == nullptr) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<FtEncodeFn>(p);
    }
    return fn;
}
// Weights: [rows, K] float32, boxes of box_rows x 32 columns, 128-byte swizzle; what lies outside reads as zero.
static bool ft_map_w(CUtensorMap* map, const void* ptr, long long rows, long long K, int box_rows) {
    cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
    cuuint64_t strides[1] = {static_cast<cuuint64_t>(K) * 4};
    cuuint32_t box[2] = {FT_K, static_cast<cuuint32_t>(box_rows)}, step[2] = {1, 1};
    return ft_encode_fn() != nullptr &&
           ft_encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(ptr), dims, strides, box, step,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// The parts of x: [3][rows][Kp] bfloat16, boxes of 3 x box_rows x 32 columns, 64-byte swizzle.
static bool ft_map_x(CUtensorMap* map, void* ptr, long long rows, long long Kp, int box_rows) {
    cuuint64_t dims[3] = {static_cast<cuuint64_t>(Kp), static_cast<cuuint64_t>(rows), 3};
    cuuint64_t strides[2] = {static_cast<cuuint64_t>(Kp) * 2, static_cast<cuuint64_t>(rows * Kp) * 2};
    cuuint32_t box[3] = {FT_K, static_cast<cuuint32_t>(box_rows), 3}, step[3] = {1, 1, 1};
    return ft_encode_fn() != nullptr &&
           ft_encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, ptr, dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int TN, bool SWIGLU>
static int launch_f32_tc(const GemmArgs& a, const CUtensorMap& map_w, const CUtensorMap& map_w2, bf16* parts, int Kp, int tiles_y,
                         cudaStream_t stream) {
    // the boxes that tiles of this call ask for: a plain product's full tiles and its last one; of experts' any (a map takes the host
    // about half a microsecond)
    FtXMaps maps_x;
    memset(&maps_x, 0, sizeof(maps_x));
    const int rest = a.M % TN, last = rest == 0 ? 3 : (rest + TN / 4 - 1) / (TN / 4) - 1;
    for (int q = 0; q < 4; ++q)
        if ((a.tile_expert != nullptr || q == last || (q == 3 && a.M >= TN)) && !ft_map_x(&maps_x.m[q], parts, a.M, Kp, (q + 1) * (TN / 4)))
            return LOCUS_ERR_UNSUPPORTED;
    auto* kernel = gemm_f32_tc_kernel<TN, SWIGLU>;
    constexpr int smem = FtShape<TN>::SMEM;
    static_assert(smem <= 227 * 1024, "shared memory");
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return static_cast<int>(e);
    static int n_sm = 0;
    if (n_sm == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            return static_cast<int>(cudaGetLastError());
    }
    const int tiles_x = ceil_div(a.N, SWIGLU ? FT_W / 2 : FT_W);
    const long long n = static_cast<long long>(tiles_x) * tiles_y * a.splits;
    if (n >= (1LL << 31)) return LOCUS_ERR_UNSUPPORTED;
    const unsigned cut_blocks = static_cast<unsigned>((static_cast<long long>(a.M) * (Kp / 8) + 255) / 256);
    f32_cut_kernel<<<cut_blocks, 256, 0, stream>>>(static_cast<const float*>(a.x), a.ldx, a.x_rows, a.x_row_div, a.K, Kp, a.M, parts);
    kernel<<<static_cast<unsigned>(n < n_sm ? n : n_sm), FT_THREADS, smem, stream>>>(map_w, map_w2, maps_x, a, tiles_x, tiles_y);
    if (a.part) gemm_f32_sum_kernel<<<dim3(ceil_div(a.N, 256), a.M), 256, 0, stream>>>(a);
    return locus_launch_status();
}

// float32 x (row stride ldx), w (and w2) [w_rows_total, K]; K and ldx multiples of 4, 16-byte aligned bases.  tn: rows of a
// tile, 64 or 128 (a grouped product's tile list has tiles of at most 64).  x_parts: scratch for the parts of the M rows,
// 3 * M * (K rounded up to a multiple of 32) bfloat16, 16-byte aligned.  The other arguments as locus_gemm_simt's.
extern "C" int locus_gemm_f32_tc(const void* x, const void* w, const void* w2, long long w_rows_total, const void* bias, int bias_dt,
                                 void* out, int out_dt, int flags, float act_param, float act_scale, const float* row_scale,
                                 const int* scale_rows, const int* x_rows, int x_row_div, int M, int N, int K, long long ldx,
                                 long long ldo, int tn, const int* tile_expert, const int* tile_row0, const int* tile_rows,
                                 const int* n_tiles, int max_tiles, void* x_parts, float* part, int splits, cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0 || ((K | ldx) & 3) != 0 || (tn != 64 && tn != 128) || w_rows_total >= (1LL << 31)) return LOCUS_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(w2) |
         reinterpret_cast<uintptr_t>(x_parts)) & 15)
        return LOCUS_ERR_UNSUPPORTED;
    const int accumulate = flags & 1, act = (flags >> 1) & 7;
    const bool swiglu = w2 != nullptr;
    if ((act == 1 && swiglu) || ((act == 2 || act == 4) && !swiglu) || act > 4 || (act == 3 && (swiglu || !(act_param > 0.f)))) return LOCUS_ERR_UNSUPPORTED;
    if ((accumulate && out_dt != LOCUS_DT_F32) || (x_rows != nullptr && x_row_div <= 0) || x_parts == nullptr) return LOCUS_ERR_UNSUPPORTED;
    if (splits < 1 || (splits > 1 && (part == nullptr || splits > 8 || swiglu || tile_expert != nullptr || M > 65535))) return LOCUS_ERR_UNSUPPORTED;
    if (tile_expert != nullptr && tn != 64) return LOCUS_ERR_UNSUPPORTED;
    const int tiles_y = tile_expert ? max_tiles : ceil_div(M, tn), Kp = ceil_div(K, FT_K) * FT_K;
    if (M == 0 || tiles_y <= 0) return 0;
    CUtensorMap map_w, map_w2;
    if (!ft_map_w(&map_w, w, w_rows_total, K, swiglu ? FT_W / 2 : FT_W)) return LOCUS_ERR_UNSUPPORTED;
    map_w2 = map_w;
    if (swiglu && !ft_map_w(&map_w2, w2, w_rows_total, K, FT_W / 2)) return LOCUS_ERR_UNSUPPORTED;
    GemmArgs a;
    a.x = x; a.w = w; a.w2 = w2; a.bias = bias; a.bias_dt = bias_dt; a.out = out; a.out_dt = out_dt; a.accumulate = accumulate;
    a.act = act; a.act_param = act_param; a.act_scale = act_scale; a.row_scale = row_scale; a.scale_rows = scale_rows;
    a.x_rows = x_rows; a.x_row_div = x_row_div; a.M = M; a.N = N; a.K = K; a.ldx = ldx; a.ldo = ldo; a.tile_expert = tile_expert;
    a.tile_row0 = tile_row0; a.tile_rows = tile_rows; a.n_tiles = n_tiles; a.w_expert_stride = 0;
    a.part = splits > 1 ? part : nullptr; a.splits = splits;
    auto* launch = tn == 64 ? (swiglu ? launch_f32_tc<64, true> : launch_f32_tc<64, false>)
                            : (swiglu ? launch_f32_tc<128, true> : launch_f32_tc<128, false>);
    return launch(a, map_w, map_w2, static_cast<bf16*>(x_parts), Kp, tiles_y, stream);
}

// Reads and clears the error word of the kernel above (0 = no bounded wait ran out).  Synchronises.
extern "C" int locus_gemm_f32_tc_error() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_f32_tc_error, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) cudaMemcpyToSymbol(g_f32_tc_error, &zero, sizeof(int));
    return v;
}
