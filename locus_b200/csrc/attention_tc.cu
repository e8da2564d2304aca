// Attention of long prompt portions on the Blackwell tensor cores (tcgen05.mma, scores and the
// weighted sums of V in tensor memory), bfloat16 queries / keys / values, softmax in float32.
//
// A block takes 128 consecutive new tokens of one request and one head.  Keys and values come in
// tiles of 128 positions through the request's block table: TMA boxes of 64 rows x 64 elements
// (pages are a multiple of 64 tokens, so a box never straddles pages; a box whose page does not
// exist is fetched from outside the tensor and arrives as zeros), three tiles of either on
// their way or in use.
//
//   MMA 1:  S[q, t] = sum_d Q[q, d] K[t, d]        (A = Q, B = K, both K-major; 128 x 128 in TMEM)
//   softmax: the thread of a query row reads its row of S (tcgen05.ld), masks (causal, window, end of the sequence), keeps
//           the running maximum and denominator (base 2), writes P = exp2(s - m) as bfloat16 over S in tensor memory
//   MMA 2:  O[q, d] += sum_t P[q, t] V[t, d]      (A = P from tensor memory, B = V read MN-major: V lies [t][d] in the
//           cache, which is the transposed operand; 128 x 128 in TMEM, ONE sum from the first tile to the last)
//   The row's thread rescales O in tensor memory (tcgen05.ld, multiply, tcgen05.st) only when the row's maximum
//   has run ahead of the reference its probabilities are formed against by more than 2^8.
//
// A tile costs the tensor cores 1,024 cycles and its exponentials as many of the special-function units, so the two have to work
// at the same time.  Two groups of four warps take the even and the odd key tiles, and three buffers of scores (with the sum of V
// all of tensor memory) let the tensor cores form scores two tiles ahead: while one group is at its exponentials the other loads
// scores and looks for maxima, and neither waits for a product.  All tiles add to one sum, against one reference maximum a row,
// which is handed from each tile's thread to the next tile's, in the other group, as soon as it is known.
// Measured, 2,048 tokens behind 8,192, 28 heads on 4: 253 us; one group of eight warps, two threads to a row, P through
// shared memory 368 (all warps in the same phase at the same time); a sum and a buffer of scores for either group 307 (each
// tile's scores waited for the group's sum before).
// Warp 0: TMA; warps 1 and 2: MMA issue (one thread each); warps 4-11: softmax and output, a thread per query row.  Head size
// 128 only (other
// sizes and pages that are not a multiple of 64 tokens go to the mma.sync kernel).
//
// Keys and values may also lie in plain rows instead of pages (rows form): two matrices [rows][kv heads * 128] in which a
// segment's keys are consecutive rows from kv_row0[segment] on (latent attention expands its heads' keys and values of a
// long portion's context that way); only the coordinates of the loads differ.  Queries and keys may then have a rotated part of
// 64 more dimensions, the keys' one row for all heads: a third 64 columns of Q and K in shared memory, two tiles of K and V
// instead of three (208 KB).  A latent mixer's portion of 1,000 tokens, 16 heads: 16.0 us, with the gather and the product that
// expands the keys 23, where the two per-head products and the attention over 576-wide latents took 178; 1,500 tokens behind 3,000:
// the whole mixer 1,660 -> 196 us, with no larger error against 64 bits (3.3e-3, 3.1e-3).
//
// Every wait on an mbarrier is bounded; when one runs out the kernel sets the module's error word,
// and every later wait of every role returns at once, so the kernel ends quickly instead of hanging.
#include <cuda.h>
#include <string.h>

#include "common.cuh"
#include "distance.cuh"
#include "mask.cuh"
#include "sink.cuh"

#define AT_HD 128        // head size
#define AT_MQ 128        // queries per block
#define AT_MK 128        // keys per tile
#define AT_HALF_BYTES (128 * 128)     // 128 rows x 64 elements: one swizzled half of an operand tile
#define AT_TILE_BYTES (2 * AT_HALF_BYTES)
#define AT_WAIT_LIMIT 200000000LL

__device__ int g_at_error = 0;

struct TcAttnArgs {
    bf16* out;
    const int* seg_q0;
    const int* seg_qn;
    const int* seg_ctx;
    const int* block_table;
    int table_stride;
    const int* kv_row0;     // rows form: a segment's first row of K and V (block_table unused); null: pages
    const int* items;
    int nh, nkv, page_tokens, window, chunk;  // (mask.cuh)
    const float* sink_val;  // with sink: a learned score per query head in its place (null: the score 0)
    int keep_first, sink;   // with a window: a request's first tokens stay in sight; one more term of score 0 in the denominator
    const float* slopes;    // distance bias per query head (distance.cuh), or null
    float scale;
    // Ranges of key tiles per block of queries (1: a block writes the result itself).  With more, a block takes
    // one range (blockIdx.z) and leaves, per query row of the step and head, its unnormalised sum, its running
    // maximum (base 2, scaled) and its denominator; attn_chunk_tc_merge_kernel adds the ranges up in ascending order.
    int n_splits;
    float* part_o;    // [row][head][split][128]
    float* part_ml;   // [row][head][split][2]
};

// Key tiles of a block of nq queries whose first sits at position p0: first the n_keep tiles of the kept first
// tokens that lie wholly in front of the window's first tile (tile j at position j * AT_MK), then the window's
// (tile j at first_tile + (j - n_keep) * AT_MK); their number, and how they are cut into ranges (the same in both
// kernels).
__device__ __forceinline__ void at_tiles(int p0, int nq, int window, int chunk, int keep_first, int n_splits, int& first_tile,
                                         int& n_keep, int& n_tiles, int& per_split) {
    const int t_hi = p0 + nq - 1;
    const int t_lo = first_key(window, chunk, p0);
    first_tile = (t_lo / AT_MK) * AT_MK;
    n_keep = (window > 0 && keep_first > 0) ? min((keep_first + AT_MK - 1) / AT_MK, first_tile / AT_MK) : 0;
    n_tiles = n_keep + (t_hi - first_tile) / AT_MK + 1;
    per_split = (n_tiles + n_splits - 1) / n_splits;
}

__device__ __forceinline__ uint32_t at_smem(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void at_bar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void at_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void at_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool at_try_wait(uint32_t bar, uint32_t parity) {
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
__device__ __forceinline__ bool at_wait(uint32_t bar, uint32_t parity, int code) {
    if (at_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (int i = 1; !at_try_wait(bar, parity); ++i) {
        if ((i & 63) == 0 && *reinterpret_cast<volatile int*>(&g_at_error) != 0) return false;   // (a trip to L2)
        if (clock64() - t0 > AT_WAIT_LIMIT) {
            atomicCAS(&g_at_error, 0, code);
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ void at_tma_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar)
        : "memory");
}
// Shared-memory operand descriptors, 128-byte swizzle.  K-major: rows of 128 bytes, 8-row groups
// 1024 bytes apart.  MN-major (the operand lies transposed): 64 elements of the M/N side are the
// contiguous 128 bytes, the next 64 are `lbo_bytes` further on, 8-row groups of the k side 1024 apart.
__device__ __forceinline__ uint64_t at_desc_k(uint32_t saddr) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((saddr & 0x3FFFF) >> 4);
    d |= static_cast<uint64_t>(1) << 16;
    d |= static_cast<uint64_t>(1024 >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}
__device__ __forceinline__ uint64_t at_desc_mn(uint32_t saddr, uint32_t lbo_bytes) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((saddr & 0x3FFFF) >> 4);
    d |= static_cast<uint64_t>(lbo_bytes >> 4) << 16;
    d |= static_cast<uint64_t>(1024 >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}
__device__ __forceinline__ void at_mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
}
// The same with A in tensor memory (lane: row; a column two elements of k).
__device__ __forceinline__ void at_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void at_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void at_ld32(uint32_t taddr, uint32_t* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,"
        "%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
}
// 2^x for x <= 0 by the special-function unit alone (exp2f adds range handling that the softmax does
// not need: a result that underflows may be zero).
__device__ __forceinline__ float at_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t at_pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

// Packed float32 pairs (one instruction for two lanes of arithmetic) and a three-way maximum: the softmax
// warps are bound by instruction issue as much as by the special-function unit.
__device__ __forceinline__ unsigned long long at_pair(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void at_unpair(unsigned long long v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long at_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long at_add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long at_mul2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float at_max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ void at_st32(uint32_t taddr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,"
        "%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
          "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
          "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
          "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}

// The weighted sum of V stays in tensor memory from a block's first key tile to its last: the MMAs of every tile add
// to it.  A row's probabilities are formed against a reference maximum that follows the row's true running maximum
// only when that has run ahead by more than 2^AT_LAG_LOG2; then, and only then, the row's sum is read, rescaled
// and written back.  Probabilities reach 2^8 at most, far inside bfloat16's and float32's range, and the quotient
// sum / denominator is the same number whatever reference it was formed with.
#define AT_LAG_LOG2 8.0f

#define AT_S 3   // tiles of scores in tensor memory: tile j's in place j % 3

// A block's barriers, in the order in which they lie in shared memory, and what is waited for before each of its steps: a barrier
// and the parity of the turn of its place.  A wait by parity cannot tell a turn from the one two further on, so whoever waits for the
// end of a turn must know that the one before it has ended, and must itself keep the one behind it from ending.
// tests/test_attention_tc_waits.py walks through every order of the roles' steps with these waits.
struct AtWait {
    int bar;
    uint32_t parity;
};
#define AT_BARS 20   // places for them
template <bool ROT>
struct AtBars {
    static constexpr int D = ROT ? 2 : 3;   // tiles of K and of V in shared memory
    static constexpr int Q_FULL = 0, K_FULL = 1, K_FREE = K_FULL + D, V_FULL = K_FREE + D, V_FREE = V_FULL + D, S_FULL = V_FREE + D,
                         P_READY = S_FULL + AT_S, DONE = P_READY + AT_S;
    // A place of the scores is free when the tile's P V is finished.  With as many places of V as of scores that is the barrier of V's
    // place; with fewer, the next tile's but one would end the turn behind on that one, which nothing keeps it from before the
    // scores are waited for.
    static constexpr int S_FREE = ROT ? DONE + 1 : V_FREE, COUNT = DONE + 1 + (ROT ? AT_S : 0);
    __host__ __device__ static constexpr AtWait full(int first, int places, int j) {
        return {first + j % places, static_cast<uint32_t>(j / places) & 1};
    }
    __host__ __device__ static constexpr AtWait free(int first, int places, int j) {   // of the tile before in tile j's place
        return {first + j % places, (static_cast<uint32_t>(j / places) & 1) ^ 1};
    }
    // the loader, before tile j's K and V; the score warp, for K and for the scores' place; the warp that sums V up, for V and the weights
    __host__ __device__ static constexpr AtWait k_place(int j) { return free(K_FREE, D, j); }
    __host__ __device__ static constexpr AtWait v_place(int j) { return free(V_FREE, D, j); }
    __host__ __device__ static constexpr AtWait k_there(int j) { return full(K_FULL, D, j); }
    __host__ __device__ static constexpr AtWait s_place(int j) { return free(S_FREE, AT_S, j); }
    __host__ __device__ static constexpr AtWait v_there(int j) { return full(V_FULL, D, j); }
    __host__ __device__ static constexpr AtWait p_there(int j) { return full(P_READY, AT_S, j); }
    // a softmax warp, for tile j's scores and for the sum that the tile before is in
    __host__ __device__ static constexpr AtWait s_there(int j) { return full(S_FULL, AT_S, j); }
    __host__ __device__ static constexpr AtWait summed(int j) { return full(V_FREE, D, j); }
    // ... and, before tile j's rows of V are touched, for the sum of the tile before in V's place (that of tile j - 3 is in when the scores
    // of tile j are there: with three places nothing is left to wait for), then for V
    static constexpr bool V_CLEAR_WAITS = ROT;
    __host__ __device__ static constexpr AtWait v_clear(int j) { return full(S_FREE, AT_S, j - D); }
    // ... and, at the end, for the last sum, by a barrier that is used once (V's place may be a turn further than a late warp's wait takes it
    // to be)
    __host__ __device__ static constexpr AtWait done(int) { return {DONE, 0}; }
};

// BIAS: a distance bias; an instance of its own (the softmax warps are bound by instruction issue).
// ROT: a rotated part (rows form).
template <bool BIAS, bool ROT>
__global__ void __launch_bounds__(384, 1)
attn_chunk_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                     const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_qr,
                     const __grid_constant__ CUtensorMap map_kr, TcAttnArgs a) {
    using B = AtBars<ROT>;
    constexpr int AT_D = B::D;
    constexpr int AT_QK_BYTES = (ROT ? 3 : 2) * AT_HALF_BYTES;      // a tile of Q or K
    extern __shared__ __align__(1024) uint8_t at_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the late tiles of a prompt see the most keys: the grid takes them first, for all heads (the heads are the
    // fast index of the grid, so that the blocks go out longest first and the last SMs to finish hold short ones)
    const int item = gridDim.y - 1 - blockIdx.y;
    const int seg = a.items[2 * item], qoff = a.items[2 * item + 1];
    if (qoff & 64) return;  // items are tiles of 64 queries; a block takes an even one and its upper neighbour
    const int h = blockIdx.x, kvh = h / (a.nh / a.nkv);
    const int nq = min(AT_MQ, a.seg_qn[seg] - qoff);
    const int row0 = a.seg_q0[seg] + qoff;
    const int p0 = a.seg_ctx[seg] + qoff;
    const int t_hi = p0 + nq - 1;
    const int t_lo = first_key(a.window, a.chunk, p0);
    const int P = a.page_tokens;
    // this block's range of the key tiles (all of them when the keys are not cut)
    int first_tile, n_keep, n_tiles_all, per_split;
    at_tiles(p0, nq, a.window, a.chunk, a.keep_first, a.n_splits, first_tile, n_keep, n_tiles_all, per_split);
    const int split = blockIdx.z;
    const int j0 = split * per_split;  // this block's first tile in the list of all
    const int n_tiles = max(0, min(per_split, n_tiles_all - j0));
    if (n_tiles == 0) return;  // the merge counts the live ranges the same way
    const int keep = a.window > 0 ? a.keep_first : 0;
    auto tile_at = [&](int j) -> int {  // first position of this block's tile j
        const int jj = j0 + j;
        return jj < n_keep ? jj * AT_MK : first_tile + (jj - n_keep) * AT_MK;
    };
    const int* table = a.kv_row0 ? nullptr : a.block_table + static_cast<size_t>(seg) * a.table_stride;

    // shared memory: Q, K[3], V[3] (each a tile of two swizzled halves), then the barriers.  That is nearly
    // all the shared memory a block can have, so the tiles start at the very base, which must be
    // 1024-byte aligned for the swizzle (checked: a block that finds it otherwise reports and leaves).
    const uint32_t base = at_smem(at_raw);
    if (base & 1023u) {
        if (threadIdx.x == 0) atomicCAS(&g_at_error, 0, 12);
        return;
    }
    const uint32_t sQ = base, sK = sQ + AT_QK_BYTES, sV = sK + AT_D * AT_QK_BYTES, bars = sV + AT_D * AT_TILE_BYTES;
    const uint32_t q_full = bars + 8 * B::Q_FULL, k_full = bars + 8 * B::K_FULL, k_free = bars + 8 * B::K_FREE, v_full = bars + 8 * B::V_FULL;
    const uint32_t v_free = bars + 8 * B::V_FREE, s_full = bars + 8 * B::S_FULL, p_ready = bars + 8 * B::P_READY, done = bars + 8 * B::DONE, s_free = bars + 8 * B::S_FREE;
    const uint32_t slot = bars + 8 * AT_BARS;
    static_assert(B::COUNT <= AT_BARS, "barriers");
    auto wait = [&](AtWait w, int code) { return at_wait(bars + 8 * w.bar, w.parity, code); };

    if (threadIdx.x == 0) {
        at_bar_init(q_full, 1);
        at_bar_init(done, 1);
        for (int b = 0; b < AT_D; ++b) {
            at_bar_init(k_full + 8 * b, 1);
            at_bar_init(k_free + 8 * b, 1);
            at_bar_init(v_full + 8 * b, 1);
            at_bar_init(v_free + 8 * b, 1);     // the tile's P V is finished
        }
        for (int b = 0; b < AT_S; ++b) {
            if (ROT) at_bar_init(s_free + 8 * b, 1);
            at_bar_init(s_full + 8 * b, 1);
            at_bar_init(p_ready + 8 * b, 4);    // one arrival per softmax warp of the group
        }
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
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(at_raw + (slot - base));
    const uint32_t tS = tmem, tO = tmem + AT_S * AT_MK;  // three S (and P over it), O: 128 columns each

    // Registers by role: of the 168 a thread that the block was launched with, what the first four warps give back goes to the
    // softmax (56 + 2 x 224 <= 3 x 168).
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp == 0) {
            uint32_t elected;
            asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
            if (elected) {
                // Q: pieces of 64 elements, rows row0 .. row0 + 127 (rows past the portion are never stored)
                const int col = h * (ROT ? AT_HD + 64 : AT_HD);
                at_expect_tx(q_full, AT_QK_BYTES);
                at_tma_2d(sQ, &map_q, col, row0, q_full);
                at_tma_2d(sQ + AT_HALF_BYTES, &map_q, col + 64, row0, q_full);
                if (ROT) at_tma_2d(sQ + 2 * AT_HALF_BYTES, &map_qr, h * 64, row0, q_full);
            }
            const long long rows_per_page = 2LL * a.nkv * P;
            const int v_shift = a.kv_row0 ? 0 : a.nkv * P;  // V rows of a page lie nkv * P rows behind its K rows
            const int col0 = a.kv_row0 ? kvh * AT_HD : 0;
            const int rows0 = a.kv_row0 ? a.kv_row0[seg] : 0;
            // Row of the pool (viewed as [pages * 2 * nkv * P][hd]) of the 64-key half hh of tile j; a half with no page, or wholly
            // outside the keys this block may see, is fetched from outside the tensor.  The lanes look up sixteen tiles at a time, sixteen
            // ahead: with a trip to the table and back before every tile the loader was what a long context waited for.
            auto look_up = [&](int j, int hh) -> int {
                const int t = tile_at(j) + 64 * hh;
                const bool seen = j < n_tiles && t <= t_hi && (t + 63 >= t_lo || t < keep);
                if (!seen) return -64;
                if (a.kv_row0) return rows0 + t;
                const int page = table[t / P];
                return page < 0 ? -64 : static_cast<int>(page * rows_per_page + static_cast<long long>(kvh) * P + t % P);
            };
            int now = look_up(lane >> 1, lane & 1), ahead = look_up(16 + (lane >> 1), lane & 1);
            auto rows_of = [&](int j) -> int2 {   // (asked for in ascending order)
                if (j > 0 && (j & 15) == 0) {
                    now = ahead;
                    ahead = look_up(j + 16 + (lane >> 1), lane & 1);
                }
                return make_int2(__shfl_sync(0xffffffffu, now, 2 * (j & 15)), __shfl_sync(0xffffffffu, now, 2 * (j & 15) + 1));
            };
            auto load = [&](bool key, int2 rows, int j) {
                const int b = j % AT_D;
                const uint32_t bar = (key ? k_full : v_full) + 8 * b;
                wait(key ? B::k_place(j) : B::v_place(j), 1);
                if (elected) {
                    const uint32_t dst = key ? sK + b * AT_QK_BYTES : sV + b * AT_TILE_BYTES;
                    const CUtensorMap* map = key ? &map_k : &map_v;
                    const int shift = key ? 0 : v_shift, ra = rows.x < 0 ? -64 : rows.x + shift, rb = rows.y < 0 ? -64 : rows.y + shift;
                    at_expect_tx(bar, key ? AT_QK_BYTES : AT_TILE_BYTES);
                    at_tma_2d(dst, map, col0, ra, bar);
                    at_tma_2d(dst + AT_HALF_BYTES, map, col0 + 64, ra, bar);
                    at_tma_2d(dst + 64 * 128, map, col0, rb, bar);
                    at_tma_2d(dst + AT_HALF_BYTES + 64 * 128, map, col0 + 64, rb, bar);
                    if (ROT && key) {
                        at_tma_2d(dst + 2 * AT_HALF_BYTES, &map_kr, 0, ra, bar);
                        at_tma_2d(dst + 2 * AT_HALF_BYTES + 64 * 128, &map_kr, 0, rb, bar);
                    }
                }
                __syncwarp();
            };
            int2 r[AT_D + 1];   // the rows of tiles j .. j + AT_D
#pragma unroll
            for (int j = 0; j < AT_D; ++j) {
                r[j] = make_int2(-64, -64);
                if (j < n_tiles) {
                    r[j] = rows_of(j);
                    load(true, r[j], j);
                }
            }
            for (int j = 0; j < n_tiles; ++j) {
                load(false, r[0], j);
                if (j + AT_D < n_tiles) {
                    r[AT_D] = rows_of(j + AT_D);
                    load(true, r[AT_D], j + AT_D);
                }
#pragma unroll
                for (int i = 0; i < AT_D; ++i) r[i] = r[i + 1];
            }
        } else if (warp < 3) {
            // Warp 1 issues the scores, warp 2 the sums of V: a thread that did both would leave the tensor cores idle while it waits
            // for one tile's weights and gives its places back.  (The whole warp walks, one thread issues: what does not depend on
            // the lane stays in uniform registers.)
            uint32_t elected;
            asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
            // f32 accumulate, bf16 x bf16, M = 128, N = 128; MMA 2 reads its B operand MN-major
            const uint32_t idesc1 = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(AT_MK >> 3) << 17) |
                                    (static_cast<uint32_t>(AT_MQ >> 4) << 24);
            const uint32_t idesc2 = idesc1 | (1u << 16);
            if (warp == 1) at_wait(q_full, 0, 5);
            for (int j = 0; j < n_tiles; ++j) {
                const int d = j % AT_D, b = j % AT_S;   // places of K and V, of the scores
                if (warp == 1) {
                    wait(B::k_there(j), 3);
                    wait(B::s_place(j), 4);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (elected) {
#pragma unroll
                        for (int ks = 0; ks < (ROT ? AT_HD + 64 : AT_HD) / 16; ++ks) {  // S = Q K^T
                            const uint32_t off = (ks >> 2) * AT_HALF_BYTES + (ks & 3) * 32;
                            at_mma(tS + b * AT_MK, at_desc_k(sQ + off), at_desc_k(sK + d * AT_QK_BYTES + off), idesc1, ks > 0);
                        }
                        at_commit(s_full + 8 * b);
                        at_commit(k_free + 8 * d);
                    }
                } else {
                    wait(B::v_there(j), 7);
                    wait(B::p_there(j), 6);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (elected) {
#pragma unroll
                        for (int ks = 0; ks < AT_MK / 16; ++ks)  // O += P V
                            at_mma_ts(tO, tS + b * AT_MK + 8 * ks, at_desc_mn(sV + d * AT_TILE_BYTES + ks * (16 * 128), AT_HALF_BYTES), idesc2,
                                      (j > 0 || ks > 0) ? 1u : 0u);
                        at_commit(v_free + 8 * d);
                        if (ROT) at_commit(s_free + 8 * b);
                        if (j == n_tiles - 1) at_commit(done);
                    }
                }
                __syncwarp();
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
        const int quarter = warp & 3, x = (warp - 4) >> 2;   // quarter of tensor memory's lanes; even or odd tiles
        const int r = quarter * 32 + lane;  // this thread's query row
        const int pq = p0 + r;              // its position
        const uint32_t lane_bits = static_cast<uint32_t>(quarter * 32) << 16;
        const float scale_log2 = a.scale * 1.4426950408889634f;
        // what a score is multiplied by behind its maximum: with a bias it is scaled when the bias is taken off
        const float mult = BIAS ? 1.0f : scale_log2;
        const unsigned long long scale2 = at_pair(mult, mult);
        const float slope = BIAS ? slope_log2(a.slopes, h) : 0.f;
        float m_run = -INFINITY, l_run = 0.f;  // the row's reference maximum (base 2, scaled); this group's part of the denominator
        bool ok = true;
        const int lo = first_key(a.window, a.chunk, pq);                    // first key this row sees ...
        const int lo_last = first_key(a.window, a.chunk, p0 + AT_MQ - 1);   // ... and the block's last row
        const uint32_t tOmine = tO + lane_bits;
        float2* ml = reinterpret_cast<float2*>(at_raw + (slot + 16 - base));   // [2][128]: what the groups' threads tell each other

        for (int j = x; j < n_tiles; j += 2) {
            const int tile0 = tile_at(j), b = j % AT_S;
            const uint32_t tSx = tS + b * AT_MK + lane_bits;
            if (!wait(B::s_there(j), 10)) ok = false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t s[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c) at_ld32(tSx + 32 * c, s[c]);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            // a key t counts for this row when lo <= t <= pq, or when it is one of the kept first tokens; only tiles
            // at an edge need the test (a tile of kept tokens lies in front of t_lo, so it is always tested)
            const bool need_mask = tile0 + AT_MK - 1 > p0 || tile0 < lo_last;
            if constexpr (BIAS) {
                // s <- s scale + slope (t - pq), two keys at a time: the first key's share (t - pq is an exact float32),
                // then a multiple of the slope per key
                const unsigned long long k2 = at_pair(scale_log2, scale_log2), sl2 = at_pair(slope, slope);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float d0 = slope * static_cast<float>(tile0 + 32 * c - pq);
                    const unsigned long long b0 = at_pair(d0, d0);
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        float u, v;
                        const unsigned long long at2 = at_pair(static_cast<float>(i), static_cast<float>(i + 1));
                        at_unpair(at_fma2(at_pair(__uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1])), k2, at_fma2(sl2, at2, b0)), u, v);
                        s[c][i] = __float_as_uint(u);
                        s[c][i + 1] = __float_as_uint(v);
                    }
                }
            }
            if (need_mask) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const int t = tile0 + 32 * c + i;
                        if (!(t <= pq && (t >= lo || t < keep))) s[c][i] = 0xff800000u;            // -inf
                    }
            }
            float mx[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                mx[c] = fmaxf(__uint_as_float(s[c][0]), __uint_as_float(s[c][1]));
#pragma unroll
                for (int i = 2; i < 32; i += 2) mx[c] = at_max3(mx[c], __uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1]));
            }
            // the reference maximum as the tile before left it, from the other group's thread of the row
            if (j > 0) {
                asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter + 4 * (x ^ 1)) : "memory");
                const float before = ml[(x ^ 1) * 128 + r].x;
                if (before != m_run) {
                    l_run *= m_run == -INFINITY ? 1.f : at_exp2(m_run - before);
                    m_run = before;
                }
            }
            const float m_new = fmaxf(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * mult, m_run);   // (the scale is positive)
            // Does the reference maximum follow?  Only when some row of the warp has run ahead of its reference by
            // more than 2^AT_LAG_LOG2 (always at a row's first key: -inf is infinitely far; -inf - -inf is not a
            // number and compares false, so a row without a key yet keeps -inf).  Then every row of the warp moves its reference
            // and rescales its sum, once the product of the tile before is in it.
            if (__any_sync(0xffffffffu, m_new - m_run > AT_LAG_LOG2)) {
                if (j > 0) {
                    if (!wait(B::summed(j - 1), 12)) ok = false;
                    const float f = m_run == -INFINITY ? 1.f : at_exp2(m_run - m_new);
                    const unsigned long long f2 = at_pair(f, f);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                    for (int c = 0; c < AT_HD; c += 32) {
                        uint32_t v[32];
                        at_ld32(tOmine + c, v);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int d = 0; d < 32; d += 2) {
                            float u, w;
                            at_unpair(at_mul2(at_pair(__uint_as_float(v[d]), __uint_as_float(v[d + 1])), f2), u, w);
                            v[d] = __float_as_uint(u);
                            v[d + 1] = __float_as_uint(w);
                        }
                        at_st32(tOmine + c, v);
                    }
                    l_run *= f;
                }
                m_run = m_new;
            }
            ml[x * 128 + r].x = m_run;
            if (j + 1 < n_tiles) asm volatile("bar.arrive %0, 64;" ::"r"(1 + quarter + 4 * x) : "memory");
            const float m_ref = m_run == -INFINITY ? 0.f : m_run;  // exp2(-inf - 0) = 0 for a row without keys so far
            const unsigned long long neg_m2 = at_pair(-m_ref, -m_ref);
            // P = exp2(s * scale - m_ref) as bfloat16 over S
            unsigned long long sum2[2] = {at_pair(0.f, 0.f), at_pair(0.f, 0.f)};
#pragma unroll
            for (int c = 0; c < 4; c += 2) {
                uint32_t pk[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    float u, v;
                    at_unpair(at_fma2(at_pair(__uint_as_float(s[c + (i >> 4)][2 * i & 31]), __uint_as_float(s[c + (i >> 4)][(2 * i & 31) + 1])),
                                      scale2, neg_m2), u, v);
                    u = at_exp2(u);
                    v = at_exp2(v);
                    sum2[i & 1] = at_add2(sum2[i & 1], at_pair(u, v));
                    pk[i] = at_pack(u, v);   // (the conversion is not on the pipe of the exponentials: integer rounding took 1 % longer)
                }
                at_st32(tSx + 16 * c, pk);
            }
            {
                float u, v;
                at_unpair(at_add2(sum2[0], sum2[1]), u, v);
                l_run += u + v;
            }
            // the last tile may hold rows of V behind the sequence's end (never written, any bit pattern): zero them
            if (tile0 + AT_MK - 1 > t_hi) {
                const int d = j % AT_D;
                if (B::V_CLEAR_WAITS && j >= AT_D && !wait(B::v_clear(j), 14)) ok = false;
                if (!wait(B::v_there(j), 11)) ok = false;
                if (tile0 + r > t_hi)
#pragma unroll
                    for (int q8 = 0; q8 < 16; ++q8)
                        *reinterpret_cast<uint4*>(at_raw + (sV - base) + d * AT_TILE_BYTES + (q8 >> 3) * AT_HALF_BYTES + r * 128 + (q8 & 7) * 16) =
                            make_uint4(0, 0, 0, 0);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            // P is written, the sum is where the MMAs may add to it: tell the MMA warp
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) at_arrive(p_ready + 8 * b);
        }
        // The last tile's reference is the larger one and that of the sum; a group writes half of the columns of its rows.  (A group
        // without a tile counts for nothing.)
        ml[x * 128 + r] = make_float2(m_run, l_run);
        if (!wait(B::done(n_tiles - 1), 13)) ok = false;
        asm volatile("bar.sync 9, 256;" ::: "memory");
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const float2 e = ml[r], o2 = ml[128 + r];
        const float m = fmaxf(e.x, o2.x);
        const float l = (e.x == -INFINITY ? 0.f : e.y * at_exp2(e.x - m)) + (o2.x == -INFINITY ? 0.f : o2.y * at_exp2(o2.x - m));
        // the sink: one more term of score 0 (the sums are relative to 2^m); with ranges, the merge adds it
        const float inv = 1.0f / (a.sink && a.n_splits == 1 ? l + sink_term2(a.sink_val, h, m) : l);
#pragma unroll 1
        for (int c = 64 * x; c < 64 * x + 64; c += 32) {
            uint32_t v[32];
            at_ld32(tOmine + c, v);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            float o[32];
#pragma unroll
            for (int d = 0; d < 32; ++d) o[d] = __uint_as_float(v[d]);
            if (!ok || r >= nq) continue;
            if (a.n_splits > 1) {
                const size_t unit = (static_cast<size_t>(row0 + r) * a.nh + h) * a.n_splits + split;
                float* po = a.part_o + unit * AT_HD + c;
#pragma unroll
                for (int d = 0; d < 32; d += 4) *reinterpret_cast<float4*>(po + d) = make_float4(o[d], o[d + 1], o[d + 2], o[d + 3]);
                if (c == 0) *reinterpret_cast<float2*>(a.part_ml + unit * 2) = make_float2(m, l);
            } else {
                bf16* dst = a.out + (static_cast<size_t>(row0 + r) * a.nh + h) * AT_HD + c;
#pragma unroll
                for (int d = 0; d < 32; d += 8) {
                    uint4 pk;
                    pk.x = at_pack(o[d] * inv, o[d + 1] * inv);
                    pk.y = at_pack(o[d + 2] * inv, o[d + 3] * inv);
                    pk.z = at_pack(o[d + 4] * inv, o[d + 5] * inv);
                    pk.w = at_pack(o[d + 6] * inv, o[d + 7] * inv);
                    *reinterpret_cast<uint4*>(dst + d) = pk;
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

#define AT_MAX_SPLITS 16

// out[row][head] = sum over the live ranges s (ascending) of o_s 2^(m_s - M) / sum of l_s 2^(m_s - M), M = max m_s.
// One thread per (query row, four adjacent dimensions) of a block of queries and a head; the loads of all ranges
// are issued together (the loops are unrolled over the most ranges there can be).
__global__ void __launch_bounds__(128) attn_chunk_tc_merge_kernel(TcAttnArgs a) {
    const int item = blockIdx.y, h = blockIdx.z;
    const int seg = a.items[2 * item], qoff = a.items[2 * item + 1];
    if (qoff & 64) return;
    const int nq = min(AT_MQ, a.seg_qn[seg] - qoff);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nq * (AT_HD / 4)) return;
    const int r = i / (AT_HD / 4), d = (i - r * (AT_HD / 4)) * 4;
    const int row = a.seg_q0[seg] + qoff + r;
    int first_tile, n_keep, n_tiles, per_split;
    at_tiles(a.seg_ctx[seg] + qoff, nq, a.window, a.chunk, a.keep_first, a.n_splits, first_tile, n_keep, n_tiles, per_split);
    const int live = (n_tiles + per_split - 1) / per_split;
    const size_t unit0 = (static_cast<size_t>(row) * a.nh + h) * a.n_splits;
    float2 ml[AT_MAX_SPLITS];
    float4 v[AT_MAX_SPLITS];
#pragma unroll
    for (int s = 0; s < AT_MAX_SPLITS; ++s) {
        ml[s] = make_float2(-INFINITY, 0.f);
        v[s] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (s < live) {
            ml[s] = *reinterpret_cast<const float2*>(a.part_ml + (unit0 + s) * 2);
            v[s] = *reinterpret_cast<const float4*>(a.part_o + (unit0 + s) * AT_HD + d);
        }
    }
    float M = -INFINITY;
#pragma unroll
    for (int s = 0; s < AT_MAX_SPLITS; ++s) M = fmaxf(M, ml[s].x);
    float L = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int s = 0; s < AT_MAX_SPLITS; ++s) {
        const float w = ml[s].x == -INFINITY ? 0.f : exp2f(ml[s].x - M);
        L += ml[s].y * w;
        acc.x += v[s].x * w;
        acc.y += v[s].y * w;
        acc.z += v[s].z * w;
        acc.w += v[s].w * w;
    }
    if (a.sink) L += sink_term2(a.sink_val, h, M);
    const float inv = 1.0f / L;
    uint2 pk;
    pk.x = at_pack(acc.x * inv, acc.y * inv);
    pk.y = at_pack(acc.z * inv, acc.w * inv);
    *reinterpret_cast<uint2*>(a.out + (static_cast<size_t>(row) * a.nh + h) * AT_HD + d) = pk;
}

// ---------------------------------------------------------------------------
typedef CUresult (*AtEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                               const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                               CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static AtEncodeFn at_encode_fn() {
    static AtEncodeFn fn = nullptr;
    if (fn == nullptr) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess) {
            fn = reinterpret_cast<AtEncodeFn>(p);
        }
    }
    return fn;
}

// rows x cols bfloat16 matrix, row stride ld elements; box = box_rows x 64 elements, 128-byte swizzle; reads
// outside the matrix give zeros.
static bool at_make_map(CUtensorMap* map, const void* ptr, long long rows, long long cols, long long ld, int box_rows) {
    AtEncodeFn fn = at_encode_fn();
    if (fn == nullptr) return false;
    cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
    cuuint32_t box[2] = {64, static_cast<cuuint32_t>(box_rows)};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The launch shared by the entry points below: `a` carries everything but the scratch of the ranges.
static int at_launch(const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v, TcAttnArgs a, int n_items,
                     int n_splits, float* part_o, float* part_ml, cudaStream_t stream, const CUtensorMap* map_qr = nullptr,
                     const CUtensorMap* map_kr = nullptr) {
    if (n_items > 65535) return LOCUS_ERR_UNSUPPORTED;
    a.n_splits = n_splits; a.part_o = part_o; a.part_ml = part_ml;
    const bool rot = map_qr != nullptr;
    const size_t smem = (rot ? 3 * 3 + 2 * 2 : 2 + 3 * 4) * AT_HALF_BYTES + 8 * AT_BARS + 16 + 2 * 128 * 8;
    auto* kernel = a.slopes != nullptr ? (rot ? attn_chunk_tc_kernel<true, true> : attn_chunk_tc_kernel<true, false>)
                                       : (rot ? attn_chunk_tc_kernel<false, true> : attn_chunk_tc_kernel<false, false>);
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    dim3 grid(a.nh, n_items, n_splits);
    kernel<<<grid, 384, smem, stream>>>(map_q, map_k, map_v, rot ? *map_qr : map_q, rot ? *map_kr : map_k, a);
    if (n_splits > 1)
        attn_chunk_tc_merge_kernel<<<dim3(AT_MQ * (AT_HD / 4) / 128, n_items, a.nh), 128, 0, stream>>>(a);
    return locus_launch_status();
}

static bool at_scratch_ok(int n_splits, const float* part_o, const float* part_ml) {
    return n_splits >= 1 && n_splits <= AT_MAX_SPLITS &&
           (n_splits == 1 || (part_o != nullptr && part_ml != nullptr &&
                              ((reinterpret_cast<uintptr_t>(part_o) | reinterpret_cast<uintptr_t>(part_ml)) & 15) == 0));
}

// q, out [T, nh * 128] bfloat16; pool: one layer's pages [n_pages][2][nkv][page_tokens][128] bfloat16;
// items: [n_items, 2] = (segment, first query of a 64-query tile), a segment's tiles in ascending order.
// Head size 128 and pages of a multiple of 64 tokens only (LOCUS_ERR_UNSUPPORTED otherwise).
// n_splits > 1: the key tiles of every block are cut into that many ranges (at most 16); part_o holds
// T * nh * n_splits * 128 floats, part_ml T * nh * n_splits * 2; a second launch merges.
extern "C" int locus_attn_chunk_tc(const void* q, long long T, const void* pool, long long n_pages, void* out,
                                   const int* seg_q0, const int* seg_qn, const int* seg_ctx, const int* block_table,
                                   int table_stride, const int* items, int n_items, int nh, int nkv, int hd,
                                   int page_tokens, int window, int chunk, float scale, int n_splits, float* part_o,
                                   float* part_ml, int keep_first, int sink, const float* sink_val,
                                   const float* slopes, cudaStream_t stream) {
    if (n_items <= 0) return 0;
    if (!at_scratch_ok(n_splits, part_o, part_ml)) return LOCUS_ERR_UNSUPPORTED;
    if (hd != AT_HD || page_tokens <= 0 || page_tokens % 64 != 0 || !mask_ok(window, chunk, keep_first)) return LOCUS_ERR_UNSUPPORTED;
    if (nh <= 0 || nkv <= 0 || nh % nkv != 0 || nh > 65535) return LOCUS_ERR_UNSUPPORTED;
    const long long pool_rows = n_pages * 2 * nkv * page_tokens;
    if (T <= 0 || n_pages <= 0 || pool_rows >= (1LL << 31) || T >= (1LL << 31)) return LOCUS_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(pool) | reinterpret_cast<uintptr_t>(out)) & 15)
        return LOCUS_ERR_UNSUPPORTED;
    CUtensorMap map_q, map_kv;
    if (!at_make_map(&map_q, q, T, static_cast<long long>(nh) * hd, static_cast<long long>(nh) * hd, AT_MQ))
        return LOCUS_ERR_UNSUPPORTED;
    if (!at_make_map(&map_kv, pool, pool_rows, hd, hd, 64)) return LOCUS_ERR_UNSUPPORTED;
    TcAttnArgs a;
    a.out = static_cast<bf16*>(out); a.seg_q0 = seg_q0; a.seg_qn = seg_qn; a.seg_ctx = seg_ctx;
    a.block_table = block_table; a.table_stride = table_stride; a.kv_row0 = nullptr; a.items = items; a.nh = nh; a.nkv = nkv;
    a.page_tokens = page_tokens; a.window = window; a.chunk = chunk; a.scale = scale;
    a.keep_first = window > 0 ? keep_first : 0; a.sink = sink ? 1 : 0; a.sink_val = sink ? sink_val : nullptr;
    a.slopes = slopes;
    return at_launch(map_q, map_kv, map_kv, a, n_items, n_splits, part_o, part_ml, stream);
}

// The rows form: k and v [rows, >= nkv * 128] bfloat16 with row strides ldk, ldv (elements, multiples of 8, 16-byte aligned
// bases); segment s's key at position t is row kv_row0[s] + t of both.  With k_rot [rows, 64] (row stride ldkr) keys have 64 more
// dimensions, the same for all heads, and queries those of q_rot [T, nh * 64]; a head's first 128 of q then lie 192 elements
// apart (its last 64 there are not read).  Otherwise as above.
extern "C" int locus_attn_chunk_tc_rows(const void* q, long long T, const void* k, long long ldk, const void* v, long long ldv,
                                        long long rows, void* out, const int* seg_q0, const int* seg_qn, const int* seg_ctx,
                                        const int* kv_row0, const int* items, int n_items, int nh, int nkv, int hd, int window,
                                        int chunk, float scale, int n_splits, float* part_o, float* part_ml, int keep_first,
                                        int sink, const float* sink_val, const float* slopes, const void* q_rot, const void* k_rot,
                                        long long ldkr, cudaStream_t stream) {
    if (n_items <= 0) return 0;
    if (!at_scratch_ok(n_splits, part_o, part_ml)) return LOCUS_ERR_UNSUPPORTED;
    if ((q_rot != nullptr) != (k_rot != nullptr) || (k_rot != nullptr && (ldkr < 64 || ldkr % 8 != 0))) return LOCUS_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(q_rot) | reinterpret_cast<uintptr_t>(k_rot)) & 15) return LOCUS_ERR_UNSUPPORTED;
    if (hd != AT_HD || kv_row0 == nullptr || !mask_ok(window, chunk, keep_first)) return LOCUS_ERR_UNSUPPORTED;
    if (nh <= 0 || nkv <= 0 || nh % nkv != 0 || nh > 65535) return LOCUS_ERR_UNSUPPORTED;
    if (T <= 0 || T >= (1LL << 31) || rows <= 0 || rows >= (1LL << 31)) return LOCUS_ERR_UNSUPPORTED;
    const long long cols = static_cast<long long>(nkv) * hd;
    if (ldk < cols || ldv < cols || ldk % 8 != 0 || ldv % 8 != 0) return LOCUS_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(out)) & 15)
        return LOCUS_ERR_UNSUPPORTED;
    CUtensorMap map_q, map_k, map_v, map_qr, map_kr;
    const long long q_cols = static_cast<long long>(nh) * (k_rot ? hd + 64 : hd);
    if (k_rot && (!at_make_map(&map_qr, q_rot, T, static_cast<long long>(nh) * 64, static_cast<long long>(nh) * 64, AT_MQ) ||
                  !at_make_map(&map_kr, k_rot, rows, 64, ldkr, 64)))
        return LOCUS_ERR_UNSUPPORTED;
    if (!at_make_map(&map_q, q, T, q_cols, q_cols, AT_MQ) ||
        !at_make_map(&map_k, k, rows, cols, ldk, 64) || !at_make_map(&map_v, v, rows, cols, ldv, 64))
        return LOCUS_ERR_UNSUPPORTED;
    TcAttnArgs a;
    a.out = static_cast<bf16*>(out); a.seg_q0 = seg_q0; a.seg_qn = seg_qn; a.seg_ctx = seg_ctx;
    a.block_table = nullptr; a.table_stride = 0; a.kv_row0 = kv_row0; a.items = items; a.nh = nh; a.nkv = nkv;
    a.page_tokens = 64; a.window = window; a.chunk = chunk; a.scale = scale;
    a.keep_first = window > 0 ? keep_first : 0; a.sink = sink ? 1 : 0; a.sink_val = sink ? sink_val : nullptr;
    a.slopes = slopes;
    return at_launch(map_q, map_k, map_v, a, n_items, n_splits, part_o, part_ml, stream, k_rot ? &map_qr : nullptr, k_rot ? &map_kr : nullptr);
}

// What a block waits for before a step of tile j (AtBars; `which` in the order of its functions): 2 * barrier + parity, -1 for
// nothing.  Host only.
extern "C" int locus_attn_tc_wait(int rot, int which, int j) {
    auto of = [&](auto bars) -> int {
        using B = decltype(bars);
        constexpr AtWait (*f[])(int) = {B::k_place, B::v_place, B::k_there, B::s_place, B::v_there, B::p_there, B::s_there, B::summed, B::v_clear, B::done};
        if (which < 0 || which >= static_cast<int>(sizeof(f) / sizeof(f[0])) || j < 0 || (f[which] == B::v_clear && (!B::V_CLEAR_WAITS || j < B::D)))
            return -1;
        const AtWait w = f[which](j);
        return 2 * w.bar + static_cast<int>(w.parity);
    };
    return rot ? of(AtBars<true>()) : of(AtBars<false>());
}

// Reads and clears the module's error word (0 = no bounded wait ran out).  Synchronises.
extern "C" int locus_attn_tc_error() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_at_error, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) cudaMemcpyToSymbol(g_at_error, &zero, sizeof(int));
    return v;
}
