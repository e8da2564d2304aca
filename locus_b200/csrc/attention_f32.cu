// Attention of prompt portions in true float32: 64 queries of one head against every key they may see, tiles of 64 keys, on
// the CUDA cores.  Heads of up to 128; larger ones run on the chunk kernel of attention.cu.
//
// Bound by the multiply-adds and, a little above them, by the shared-memory reads that feed them: a thread owns 8 queries x
// 4 keys of the scores and then 8 queries x 8 dimensions of the output, so that 12 16-byte reads feed 64 paired
// multiply-adds in both products (pairs of dimensions: the scores' are halves of one sum, the output's two outputs).  The
// 16 threads of a query's row share a half-warp in both, so the softmax's maxima and sums cross lanes only and the
// weights go from the one product to the other through rows that a warp writes and reads by itself -- each twice, as the
// pairs want them, in the buffer that held the keys.  K and V are copied asynchronously (rows of keys 4 floats longer, so
// that 8 of them meet in no bank); two blocks of 100 KB share an SM and hide each other's copies.
// Measured: 512 tokens behind 1,500 others, 16 heads of 128: 274 us in two ranges (27 TFLOP/s) where the kernel of 16-query
// tiles with scalar loads took 1,563 to 1,859 us; with every warp working out its rows' places by itself 372.  A portion of 2 / 16
// tokens behind none 7.0 / 7.8 us (13.5 / 22.7 with 16-query tiles; 17.8 / 19.1 when all 64 rows of a tile were worked on).
//
// Mask, window with kept first tokens, chunks, sink and distance bias as in attention.cu; keys outside a tile's range are
// zeros, never what the pages hold.  A step with few tiles cuts the keys into n_splits ranges (grid z) whose unnormalised
// sums, maxima and denominators a second kernel merges in ascending order.
#include "common.cuh"
#include "distance.cuh"
#include "key_tiles.cuh"
#include "sink.cuh"
#include "walk.cuh"

#define FQ 64
#define F32_MAX_SPLITS 16

struct F32AttnArgs {
    const float* q;           // [T, nh * hd]
    const float* pool;        // this layer's pages [n_pages][2][nkv][page_tokens][hd]
    float* out;               // [T, nh * hd]
    const int* seg_q0;
    const int* seg_qn;
    const int* seg_ctx;
    const int* block_table;
    int table_stride;
    const int* items;         // [n_items, 2] (segment, first query of a 64-query tile within it)
    int nh, nkv, hd, page_tokens, window, chunk, keep_first, sink;
    const float* sink_val;
    const float* slopes;
    float scale;
    int n_splits;
    float* part_o;            // [item][head][split][FQ][hd]
    float* part_ml;           // [item][head][split][FQ][2]
};

// The weight of a key that a query must not see: a pair of -0, which no exponential is.  Its value takes no part in the sum, so
// that one that is not finite reaches nobody who does not see it (as a weight of 0 it would: 0 * inf).
static constexpr f2 HIDDEN = 0x8000000080000000ull;
template <int N>
struct Int {
    static constexpr int value = N;
};

// HD: the head size that the tiles are laid out for (hd <= HD; dimensions behind hd are zeros).
template <int HD>
__global__ void __launch_bounds__(128, 2) attn_chunk_f32_kernel(F32AttnArgs a) {
    constexpr int LD = HD + 4, DP = HD / 32;   // DP: pairs of dimensions of a thread's output
    static_assert(DP == 1 || DP == 2 || DP == 4, "heads of 32, 64 or 128");
    constexpr int KROWS = KEY_TILE * LD > KEY_TILE * KEY_TILE * 2 ? KEY_TILE * LD : KEY_TILE * KEY_TILE * 2;
    extern __shared__ __align__(16) float f32a_smem[];
    __shared__ long long rows_at[2][KEY_TILE];   // of a tile's keys in the pool, by the tile's parity; -1: not there
    float* sq = f32a_smem;         // [FQ][LD]
    float* sk = sq + FQ * LD;      // [KEY_TILE][LD]; then the weights, [FQ][KEY_TILE] pairs
    float* sv = sk + KROWS;        // [KEY_TILE][HD]
    f2* sp = reinterpret_cast<f2*>(sk);

    // the late tiles of a prompt see the most keys: the grid takes them first, for all heads (its fast index)
    const int item = gridDim.y - 1 - blockIdx.y, h = blockIdx.x, split = blockIdx.z;
    const int seg = a.items[2 * item], qoff = a.items[2 * item + 1];
    const int kvh = h / (a.nh / a.nkv), hd = a.hd, P = a.page_tokens;
    const int nq = min(FQ, a.seg_qn[seg] - qoff);
    const int row0 = a.seg_q0[seg] + qoff, p0 = a.seg_ctx[seg] + qoff;
    const int* table = a.block_table + static_cast<size_t>(seg) * a.table_stride;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, tx = tid & 15, ty = tid >> 4;
    const int t_hi = p0 + nq - 1, t_lo = first_key(a.window, a.chunk, p0), lo_last = first_key(a.window, a.chunk, t_hi);
    const int kept = a.window > 0 ? min(a.keep_first, t_lo) : 0;
    int first_tile, n_all, kept_tiles;
    item_tiles(p0, nq, a.window, a.chunk, a.keep_first, first_tile, n_all, kept_tiles);
    const int per_split = (n_all + a.n_splits - 1) / a.n_splits, first_idx = split * per_split;
    const int n_tiles = min(per_split, n_all - first_idx);
    if (n_tiles <= 0) return;   // (the merge counts the live ranges the same way)

    if (hd < HD) {   // dimensions that no copy fills
        for (int i = tid; i < (FQ + KEY_TILE) * (HD - hd); i += 128) {
            const int r = i / (HD - hd), d = hd + i % (HD - hd);
            (r < FQ ? sq + r * LD : sv + (r - FQ) * HD)[d] = 0.f;
        }
    }
    // Copies: HD / 4 lanes to a row, of 16 bytes each.  Where the rows of a tile's keys lie is worked out by a thread a row, a tile ahead
    // (by every warp for its own rows, one row after the other, a tile waited 4 us for two divisions and a table read a row).
    constexpr int RL = HD / 4, RW = 32 / RL, RI = KEY_TILE / (4 * RW);   // lanes of a row, rows of a warp's copy, copies of a warp
    const int cl = (lane % RL) * 4, rl = warp * RW + lane / RL;
    const size_t v_off = static_cast<size_t>(a.nkv) * P * hd;
    auto place = [&](int it) {
        if (tid >= KEY_TILE || it >= n_tiles) return;
        const int t = tile_pos(first_idx + it, first_tile, kept_tiles) + tid;
        long long at = -1;
        if ((t >= t_lo || t < kept) && t <= t_hi)
            at = (static_cast<long long>(table[t / P]) * 2 * a.nkv + kvh) * P * hd + static_cast<long long>(t % P) * hd;
        rows_at[it & 1][tid] = at;
    };
    place(0);
    if (cl < hd)
        for (int r = rl; r < FQ; r += 4 * RW) {
            const bool live = r < nq;
            walk_copy<16>(sq + r * LD + cl, a.q + (static_cast<size_t>(row0 + (live ? r : 0)) * a.nh + h) * hd + cl, live);
        }
    __syncthreads();
    auto copy_tile = [&](int it) {
        long long at[RI];
#pragma unroll
        for (int i = 0; i < RI; ++i) at[i] = rows_at[it & 1][rl + 4 * RW * i];
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            float* dst = sk + (rl + 4 * RW * i) * LD + cl;
            if (cl < hd) walk_copy<16>(dst, a.pool + (at[i] < 0 ? 0 : at[i] + cl), at[i] >= 0);
            else *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);   // (the weights of the last tile lay here)
        }
        walk_commit();
#pragma unroll
        for (int i = 0; i < RI; ++i)
            if (cl < hd) walk_copy<16>(sv + (rl + 4 * RW * i) * HD + cl, a.pool + (at[i] < 0 ? 0 : at[i] + v_off + cl), at[i] >= 0);
        walk_commit();
    };
    const float slope = slope_of(a.slopes, h);
    f2 o[8][DP];
    float m[8], l[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int d = 0; d < DP; ++d) o[i][d] = 0;
    }
    const int n_rows = (nq - ty + 7) >> 3;   // (of this thread's queries ty, ty + 8, .. those that are there)
    // NI: the eights of queries that are worked on.  (A lone tile takes as long as its instructions: a portion of up to 16 queries would
    // otherwise pay for 64.)
    auto walk_tiles = [&](auto eights) {
        constexpr int NI = decltype(eights)::value;
        for (int it = 0; it < n_tiles; ++it) {
            const int tile0 = tile_pos(first_idx + it, first_tile, kept_tiles);
            copy_tile(it);
            place(it + 1);
            walk_wait<1>();
            __syncthreads();
            f2 s2[NI][4];
#pragma unroll
            for (int i = 0; i < NI; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s2[i][j] = 0;
#pragma unroll 4
            for (int d = 0; d < HD; d += 4) {
                ulonglong2 x[NI];
#pragma unroll
                for (int i = 0; i < NI; ++i) x[i] = *reinterpret_cast<const ulonglong2*>(sq + (ty + 8 * i) * LD + d);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(sk + (tx + 16 * j) * LD + d);
#pragma unroll
                    for (int i = 0; i < NI; ++i) s2[i][j] = f2_fma(x[i].x, k.x, s2[i][j]);
#pragma unroll
                    for (int i = 0; i < NI; ++i) s2[i][j] = f2_fma(x[i].y, k.y, s2[i][j]);
                }
            }
            __syncthreads();   // nobody reads the keys any more: the weights take their place
            const bool need_mask = tile0 + KEY_TILE - 1 > p0 || tile0 < lo_last;
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int p = p0 + ty + 8 * i;
                float s[4], mx = m[i];
                bool hid[4];
                const int lo = first_key(a.window, a.chunk, p);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int t = tile0 + tx + 16 * j;
                    float e, f;
                    f2_unpack(s2[i][j], e, f);
                    s[j] = fmaf(slope, static_cast<float>(t - p), (e + f) * a.scale);
                    hid[j] = need_mask && !(t <= p && (t >= lo || t < a.keep_first));
                    if (hid[j]) s[j] = -INFINITY;
                    mx = fmaxf(mx, s[j]);
                }
#pragma unroll
                for (int b = 1; b < 16; b <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, b));
                const float base = mx == -INFINITY ? 0.f : mx;   // (no key seen yet: the weights are exp(-inf) = 0)
                const float alpha = expf(m[i] - base);           // exp(-inf) = 0 on the first live tile
                float sum = 0.f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float e = expf(s[j] - base);
                    sum += e;
                    sp[(ty + 8 * i) * KEY_TILE + tx + 16 * j] = hid[j] ? HIDDEN : f2_pack(e, e);
                }
                m[i] = mx;
                l[i] = l[i] * alpha + sum;   // (this thread's keys; the row's sixteen meet at the end)
                const f2 al = f2_pack(alpha, alpha);
#pragma unroll
                for (int d = 0; d < DP; ++d) o[i][d] = f2_mul(o[i][d], al);
            }
            walk_wait<0>();
            __syncthreads();   // the values are there for all warps
            auto weigh = [&](auto masked) {
                constexpr bool MASKED = decltype(masked)::value != 0;
                const int end = MASKED ? min(KEY_TILE, t_hi - tile0 + 1) : KEY_TILE;   // (behind it every key is hidden from every query)
#pragma unroll 2
                for (int k = 0; k < end; k += 2) {
                    f2 v[2][DP];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const float* vr = sv + (k + u) * HD;
                        if constexpr (DP == 1) {
                            v[u][0] = *reinterpret_cast<const f2*>(vr + 2 * tx);
                        } else {
#pragma unroll
                            for (int d = 0; d < DP / 2; ++d) {
                                const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(vr + 64 * d + 4 * tx);
                                v[u][2 * d] = w.x;
                                v[u][2 * d + 1] = w.y;
                            }
                        }
                    }
#pragma unroll
                    for (int i = 0; i < NI; ++i) {
                        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(sp + (ty + 8 * i) * KEY_TILE + k);
                        if (!MASKED || w.x != HIDDEN)
#pragma unroll
                            for (int d = 0; d < DP; ++d) o[i][d] = f2_fma(w.x, v[0][d], o[i][d]);
                        if (!MASKED || w.y != HIDDEN)
#pragma unroll
                            for (int d = 0; d < DP; ++d) o[i][d] = f2_fma(w.y, v[1][d], o[i][d]);
                    }
                }
            };
            if (need_mask) weigh(Int<1>());
            else weigh(Int<0>());
            __syncthreads();   // nobody reads the weights and the values any more
        }
    };
    if (nq <= 16) walk_tiles(Int<2>());
    else if (nq <= 32) walk_tiles(Int<4>());
    else walk_tiles(Int<8>());
    const size_t unit = (static_cast<size_t>(item) * a.nh + h) * a.n_splits + split;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float sum = l[i];
#pragma unroll
        for (int b = 1; b < 16; b <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, b);
        if (i >= n_rows) continue;
        const int r = ty + 8 * i;
        const bool whole = a.n_splits == 1;
        const float inv = whole ? 1.0f / (a.sink ? sum + sink_term(a.sink_val, h, m[i]) : sum) : 1.0f;
        float* dst = whole ? a.out + (static_cast<size_t>(row0 + r) * a.nh + h) * hd : a.part_o + (unit * FQ + r) * hd;
#pragma unroll
        for (int d = 0; d < DP; ++d) {
            const int at = DP == 1 ? 2 * tx : 64 * (d >> 1) + 4 * tx + 2 * (d & 1);
            float e, f;
            f2_unpack(o[i][d], e, f);
            if (at < hd) *reinterpret_cast<float2*>(dst + at) = make_float2(e * inv, f * inv);
        }
        if (!whole && tx == 0) *reinterpret_cast<float2*>(a.part_ml + (unit * FQ + r) * 2) = make_float2(m[i], sum);
    }
}

// One thread per (query, four dimensions): the ranges' sums in ascending order.
__global__ void __launch_bounds__(128) attn_chunk_f32_merge_kernel(F32AttnArgs a) {
    const int item = blockIdx.y, h = blockIdx.z, hd = a.hd;
    const int seg = a.items[2 * item], qoff = a.items[2 * item + 1];
    const int nq = min(FQ, a.seg_qn[seg] - qoff);
    const int i = blockIdx.x * 128 + threadIdx.x, r = i / (hd >> 2), d = (i % (hd >> 2)) * 4;
    if (r >= nq) return;
    int first_tile, n_tiles, kept_tiles;
    item_tiles(a.seg_ctx[seg] + qoff, nq, a.window, a.chunk, a.keep_first, first_tile, n_tiles, kept_tiles);
    const int per_split = (n_tiles + a.n_splits - 1) / a.n_splits, live = (n_tiles + per_split - 1) / per_split;
    const size_t unit0 = (static_cast<size_t>(item) * a.nh + h) * a.n_splits;
    float M = -INFINITY;
    for (int s = 0; s < live; ++s) M = fmaxf(M, a.part_ml[((unit0 + s) * FQ + r) * 2]);
    float L = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < live; ++s) {
        const float2 ml = *reinterpret_cast<const float2*>(a.part_ml + ((unit0 + s) * FQ + r) * 2);
        const float w = ml.x == -INFINITY ? 0.f : expf(ml.x - M);
        const float4 v = *reinterpret_cast<const float4*>(a.part_o + ((unit0 + s) * FQ + r) * hd + d);
        L = fmaf(ml.y, w, L);
        acc.x = fmaf(v.x, w, acc.x);
        acc.y = fmaf(v.y, w, acc.y);
        acc.z = fmaf(v.z, w, acc.z);
        acc.w = fmaf(v.w, w, acc.w);
    }
    const float inv = 1.0f / (a.sink ? L + sink_term(a.sink_val, h, M) : L);
    *reinterpret_cast<float4*>(a.out + (static_cast<size_t>(a.seg_q0[seg] + qoff + r) * a.nh + h) * hd + d) =
        make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
}

template <int HD>
static int launch(const F32AttnArgs& a, int n_items, cudaStream_t stream) {
    constexpr int LD = HD + 4;
    constexpr int KROWS = KEY_TILE * LD > KEY_TILE * KEY_TILE * 2 ? KEY_TILE * LD : KEY_TILE * KEY_TILE * 2;
    constexpr size_t smem = sizeof(float) * (FQ * LD + KROWS + KEY_TILE * HD);
    const cudaError_t e = cudaFuncSetAttribute(attn_chunk_f32_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    attn_chunk_f32_kernel<HD><<<dim3(a.nh, n_items, a.n_splits), 128, smem, stream>>>(a);
    if (a.n_splits > 1) attn_chunk_f32_merge_kernel<<<dim3((FQ * (a.hd >> 2) + 127) / 128, n_items, a.nh), 128, 0, stream>>>(a);
    return locus_launch_status();
}

// items: [n_items, 2] = (segment, first query of a 64-query tile).  n_splits > 1: part_o holds n_items * nh * n_splits * 64 *
// hd floats, part_ml n_items * nh * n_splits * 128.
extern "C" int locus_attn_chunk_f32(const float* q, const float* pool, float* out, const int* seg_q0, const int* seg_qn,
                                    const int* seg_ctx, const int* block_table, int table_stride, const int* items, int n_items,
                                    int nh, int nkv, int hd, int page_tokens, int window, int chunk, float scale, int n_splits,
                                    float* part_o, float* part_ml, int keep_first, int sink, const float* sink_val,
                                    const float* slopes, cudaStream_t stream) {
    if (n_items <= 0) return 0;
    if (nh <= 0 || nkv <= 0 || nh % nkv != 0 || nh > 65535 || hd <= 0 || hd % 16 != 0 || hd > 128 || page_tokens <= 0 ||
        n_items > 65535 || !mask_ok(window, chunk, keep_first))
        return LOCUS_ERR_UNSUPPORTED;
    if (n_splits < 1 || n_splits > F32_MAX_SPLITS || (n_splits > 1 && (part_o == nullptr || part_ml == nullptr)) ||
        ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(pool) | reinterpret_cast<uintptr_t>(out) |
          reinterpret_cast<uintptr_t>(part_o) | reinterpret_cast<uintptr_t>(part_ml)) & 15))
        return LOCUS_ERR_UNSUPPORTED;
    F32AttnArgs a;
    a.q = q; a.pool = pool; a.out = out; a.seg_q0 = seg_q0; a.seg_qn = seg_qn; a.seg_ctx = seg_ctx; a.block_table = block_table;
    a.table_stride = table_stride; a.items = items; a.nh = nh; a.nkv = nkv; a.hd = hd; a.page_tokens = page_tokens;
    a.window = window; a.chunk = chunk; a.keep_first = window > 0 ? keep_first : 0; a.sink = sink;
    a.sink_val = sink ? sink_val : nullptr; a.slopes = slopes; a.scale = scale; a.n_splits = n_splits; a.part_o = part_o;
    a.part_ml = part_ml;
    if (hd <= 32) return launch<32>(a, n_items, stream);
    if (hd <= 64) return launch<64>(a, n_items, stream);
    return launch<128>(a, n_items, stream);
}
