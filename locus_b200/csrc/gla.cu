// Gated linear attention: per request and head a matrix state S [d, dv] (float32, in the request's state slot, zero when
// the request opens) whose rows -- one per key channel -- decay each by a factor of their own at every token:
//
//     S_t = diag(a_t) S_(t-1) + k_t v_t^T,      o_t = S_t^T q_t * q_scale,
//
// with a_t [d] in (0, 1) per token and head.  Everything is float32; q, k, v and the decays are columns of float32 row
// matrices given by pointer, row stride and offset.  The decays travel as c = 1 - a and a row is decayed as S - c S: a
// channel that forgets slowly has a within a few float32 spacings of 1, so that a itself would carry its rate 1 - a
// with a relative error of 1e-4 and more, which a few hundred tokens turn into as much in the state; c keeps the rate
// to float32's own precision.
//
//   gla_decay   c = 1 - sigmoid(z)^(1 / tau) = -expm1(-softplus(-z) / tau) in place over rows of logits z (softplus in its
//               stable form max(x, 0) + log1p(exp(-|x|)); no fast-math)
//   gla_walk    for portions.  A block of eight warps owns 16 columns of one head's state for one request and walks the
//               request's new tokens in order, the state in registers (walk.cuh says which lane holds what).  What bounds
//               a walk is not the recurrence -- two dependent multiply-adds a token -- but its operands: with each warp
//               fetching a token ahead by itself a token took 700 ns behind a product that had left the operands in
//               DRAM and the far L2 (2,048 tokens of 16 heads of 128 x 128: 1,433 us inside the mixer).  So 16 tokens
//               of q, k and the decays are copied into shared memory together, asynchronously, a tile ahead, by all
//               warps for all, and the read-outs of eight tokens cross the lanes together: 259 us alone (745 before, the operands
//               in L2) and about as long inside the mixer, whose pass went from 1,613 to 428 us.
//   gla_tokens  for steps of few tokens a request (decoding): 16 columns of a head and 8 groups of rows to a block, so that
//               a row of the state is read and written in whole sectors (64 requests: 46 -> 24 us).
//
//   gla_chunk   for long portions of heads of 128 channels: sixteen tokens together, as matrix products.  With C_i = 1 - a_0 .. a_i and
//               R_j = 1 - a_(j+1) .. a_15 within the sixteen (formed from the c by C <- C + c - C c, so that a slow channel
//               keeps its rate),
//                   o_i = ((1 - C_i) q_i) . S + sum_(j <= i) A_ij v_j,   A_ij = sum_d q_id k_jd a_(j+1)d .. a_id,
//                   S  <- S - C_15 S + sum_j ((1 - R_j) k_j) v_j^T.
//               Everything but the last product's sum and the reading of S is the same for all columns of a head and for all tokens
//               at once: gla_chunk_prep forms it, in three bfloat16 parts (chunk_mma.cuh).  What remains of the walk is a state in
//               the registers of eight warps, sixteen channels each, 24 MMAs a warp for sixteen tokens (36 of one), and sums
//               over the warps, which nothing waits for: the chain from chunk to chunk is one multiply-add.
//               Bound by the latency of a chunk's chain of loads, cuts and MMAs, 1,320 cycles with two warps a scheduler.  Measured,
//               2,048 tokens of 16 heads of 128 x 128: 254 -> 129 us (26 of them gla_chunk_prep), eight requests of 256 178 -> 100,
//               64 of 64 437 -> 295, one of 64 12.1 -> 12.4 (of 32 9.4 / 11.1; kernels.chunks_pay draws the line); the error against
//               64 bits 4.3e-7 -> 2.0e-7 of the read-outs' norm, of the state 4.4e-7 -> 1.3e-7.  Two chunks to a turn, one block an
//               SM: 134 and 135 us.
//
// The order of every sum is fixed by d and by the kernel.
#include "common.cuh"
#include "walk.cuh"
#include "chunk_mma.cuh"

struct GlaArgs {
    const float* q;
    const float* k;
    const float* v;
    const float* a;       // 1 - decay
    float* state;
    const int* state_slots;
    const int* seg_q0;
    const int* seg_qn;
    float* out;           // [T, ldo]: head h's columns start at h * dv
    long long slot_stride;
    int ldq, off_q, ldk, off_k, ldv, off_v, lda, off_a, ldo;
    int H, d, dv;
    float q_scale;
};

// A request of few tokens in a walk's block of 256 threads: 32 columns from col0 on x 8 groups of R consecutive rows (d <= 8 R), the
// sums of a column as gla_tokens_kernel below takes them (which as an instance of this function ran 7 to 11 % longer).
// part: [4][16] for either half of the columns.
template <int R>
__device__ __forceinline__ void gla_few(const GlaArgs& a, int seg, int h, int col0, float (*ops)[8 * R], float (*part)[16]) {
    constexpr int DP = 8 * R;
    const int tid = threadIdx.x, half = tid >> 7, rg = (tid & 127) >> 4, c = tid & 15, wid = (tid & 127) >> 5;
    const int col = col0 + 16 * half + c;
    const int qn = a.seg_qn[seg], q0 = a.seg_q0[seg];
    const int d = a.d, dv = a.dv;
    const bool col_ok = col < dv;
    float* S = a.state + static_cast<size_t>(a.state_slots[seg]) * a.slot_stride + static_cast<size_t>(h) * d * dv;
    part += 4 * half;
    float s[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int r = rg * R + i;
        s[i] = (r < d && col_ok) ? S[static_cast<size_t>(r) * dv + col] : 0.f;
    }
    for (int t = 0; t < qn; ++t) {
        const size_t row = static_cast<size_t>(q0 + t);
        const float vv = col_ok ? a.v[row * a.ldv + a.off_v + h * dv + col] : 0.f;
        for (int r = tid; r < DP; r += 256) {
            ops[0][r] = r < d ? a.q[row * a.ldq + a.off_q + h * d + r] : 0.f;
            ops[1][r] = r < d ? a.k[row * a.ldk + a.off_k + h * d + r] : 0.f;
            ops[2][r] = r < d ? a.a[row * a.lda + a.off_a + h * d + r] : 0.f;
        }
        __syncthreads();
        float o0 = 0.f, o1 = 0.f;
#pragma unroll
        for (int i = 0; i < R; i += 4) {
            const float4 qv = *reinterpret_cast<const float4*>(&ops[0][rg * R + i]);
            const float4 kv = *reinterpret_cast<const float4*>(&ops[1][rg * R + i]);
            const float4 av = *reinterpret_cast<const float4*>(&ops[2][rg * R + i]);
            s[i] = fmaf(kv.x, vv, fmaf(-av.x, s[i], s[i]));
            s[i + 1] = fmaf(kv.y, vv, fmaf(-av.y, s[i + 1], s[i + 1]));
            s[i + 2] = fmaf(kv.z, vv, fmaf(-av.z, s[i + 2], s[i + 2]));
            s[i + 3] = fmaf(kv.w, vv, fmaf(-av.w, s[i + 3], s[i + 3]));
            o0 = fmaf(s[i], qv.x, o0);
            o1 = fmaf(s[i + 1], qv.y, o1);
            o0 = fmaf(s[i + 2], qv.z, o0);
            o1 = fmaf(s[i + 3], qv.w, o1);
        }
        float o = o0 + o1;
        o += __shfl_xor_sync(0xffffffffu, o, 16);
        if ((tid & 31) < 16) part[wid][c] = o;
        __syncthreads();   // (also: nobody reads the operands any more)
        if (rg == 0 && col_ok)
            a.out[row * a.ldo + h * dv + col] = ((part[0][c] + part[1][c]) + (part[2][c] + part[3][c])) * a.q_scale;
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int r = rg * R + i;
        if (r < d && col_ok) S[static_cast<size_t>(r) * dv + col] = s[i];
    }
}

#define GL_STAGES 2   // (three: two blocks an SM instead of three, 1,390 us for eight requests of 2,048 tokens, not 1,290)
#define GL_TT 16   // tokens of a tile

// RPL: rows of a column that a lane keeps, of two columns (d <= 32 RPL).  VEC: the rows of q, k and a of a head start on
// 16-byte boundaries and d is a multiple of 4, so four rows are one copy.  MIXED: requests of up to `few` tokens are taken token by
// token.
template <int RPL, bool VEC, bool MIXED>
__global__ void __launch_bounds__(32 * WALK_WARPS, RPL > 4 ? 2 : 3) gla_walk_kernel(const GlaArgs a, int col_blocks, int few) {
    constexpr int DP = 32 * RPL, CB = WALK_CW * WALK_WARPS, TT = GL_TT, TILE = TT * (3 * DP + 2 * CB), NT = 32 * WALK_WARPS;
    constexpr int RV = RPL < 4 ? RPL : 4;                // rows of a load
    extern __shared__ __align__(16) float walk_smem[];   // [GL_STAGES][q, k, a: [TT][DP]; v: [TT][CB], every value twice]
    __shared__ float read[2][TT][CB];                    // a tile's read-outs, by the tile's parity
    pdl_entry();
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int seg = blockIdx.y, h = blockIdx.x / col_blocks, col0 = (blockIdx.x % col_blocks) * CB;
    const int qn = a.seg_qn[seg], q0 = a.seg_q0[seg];
    if (qn <= 0) return;
    static_assert(NT == 256 && CB == 16, "gla_few takes the columns of two blocks");
    if (MIXED && qn <= few) {   // a request of few tokens beside portions: every other block does two blocks' columns
        if ((blockIdx.x % col_blocks) & 1) return;
        float (*part)[16] = reinterpret_cast<float (*)[16]>(walk_smem + 3 * DP);
        if (RPL == 2 && a.d <= 32) gla_few<4>(a, seg, h, col0, reinterpret_cast<float (*)[32]>(walk_smem), part);
        else gla_few<4 * RPL>(a, seg, h, col0, reinterpret_cast<float (*)[DP]>(walk_smem), part);
        return;
    }
    const int d = a.d, dv = a.dv, wc = wid * WALK_CW;
    float* S = a.state + static_cast<size_t>(a.state_slots[seg]) * a.slot_stride + static_cast<size_t>(h) * d * dv;

    // rows d .. DP of the tiles are never copied: they stay zero, and so do the state's rows there
    if (d < DP)
        for (int i = tid; i < GL_STAGES * TT * 3 * (DP - d); i += NT) {
            const int row = i / (DP - d), r = d + i % (DP - d);
            walk_smem[(row / (3 * TT)) * TILE + (row % (3 * TT)) * DP + r] = 0.f;
        }
    const float* src[3] = {a.q + a.off_q + h * d, a.k + a.off_k + h * d, a.a + a.off_a + h * d};
    const int ld[3] = {a.ldq, a.ldk, a.lda};
    const float* vsrc = a.v + a.off_v + h * dv + col0;
    auto fetch = [&](int tile) {   // a tile's operands into its buffer; tokens behind the last one are zeros
        float* buf = walk_smem + (tile % GL_STAGES) * TILE;
#pragma unroll
        for (int w = 0; w < 3; ++w)
#pragma unroll
            for (int i = 0; i < TT / WALK_WARPS; ++i) {
                const int t = wid + i * WALK_WARPS, tok = tile * TT + t;
                const bool live = tok < qn;
                const float* row = src[w] + static_cast<size_t>(q0 + (live ? tok : 0)) * ld[w];
                float* dst = buf + (w * TT + t) * DP;
                if (VEC) {
                    for (int r = 4 * lane; r < d; r += 128) walk_copy<16>(dst + r, row + r, live);
                } else {
                    for (int r = lane; r < d; r += 32) walk_copy<4>(dst + r, row + r, live);
                }
            }
        for (int i = tid; i < 2 * TT * CB; i += NT) {
            const int t = i / (2 * CB), c = (i % (2 * CB)) >> 1, tok = tile * TT + t;
            const bool live = tok < qn && col0 + c < dv;
            walk_copy<4>(buf + 3 * TT * DP + i, vsrc + (live ? static_cast<size_t>(q0 + tok) * a.ldv + c : 0), live);
        }
    };
    auto read_out = [&](int tile) {   // the read-outs of a tile that all warps have left
        for (int i = tid; i < TT * CB; i += NT) {
            const int t = i / CB, c = i % CB, tok = tile * TT + t;
            if (tok < qn && col0 + c < dv)
                a.out[static_cast<size_t>(q0 + tok) * a.ldo + h * dv + col0 + c] = read[tile & 1][t][c] * a.q_scale;
        }
    };
    const int n_tiles = (qn + TT - 1) / TT;
#pragma unroll
    for (int i = 0; i < GL_STAGES - 1; ++i) {
        if (i < n_tiles) fetch(i);
        walk_commit();
    }
    auto row_of = [&](int i) { return 128 * (i / RV) + RV * lane + (i % RV); };
    f2 s[WALK_CW][RPL / 2];
#pragma unroll
    for (int c = 0; c < WALK_CW; ++c)
#pragma unroll
        for (int i = 0; i < RPL / 2; ++i) {
            const int r = row_of(2 * i), col = col0 + wc + c;
            s[c][i] = f2_pack((r < d && col < dv) ? S[static_cast<size_t>(r) * dv + col] : 0.f,
                              (r + 1 < d && col < dv) ? S[static_cast<size_t>(r + 1) * dv + col] : 0.f);
        }
    const int mine = walk_sum_index<16>(lane);   // the value (token, column) of eight tokens that this lane ends up with
    for (int tile = 0; tile < n_tiles; ++tile) {
        walk_wait<GL_STAGES - 2>();
        __syncthreads();   // the tile is there for all warps, and nobody reads the buffer that is filled next
        if (tile + GL_STAGES - 1 < n_tiles) fetch(tile + GL_STAGES - 1);
        walk_commit();
        if (tile > 0) read_out(tile - 1);
        const float* buf = walk_smem + (tile % GL_STAGES) * TILE;
        struct Ops {
            f2 q[RPL / 2], k[RPL / 2], a[RPL / 2], v[WALK_CW];
        };
        auto load = [&](Ops& x, int t) {
            const float* qp = buf + t * DP + RV * lane;
#pragma unroll
            for (int b = 0; b < RPL / RV; ++b) {
                if constexpr (RV == 4) {
                    const ulonglong2 q4 = *reinterpret_cast<const ulonglong2*>(qp + 128 * b);
                    const ulonglong2 k4 = *reinterpret_cast<const ulonglong2*>(qp + TT * DP + 128 * b);
                    const ulonglong2 a4 = *reinterpret_cast<const ulonglong2*>(qp + 2 * TT * DP + 128 * b);
                    x.q[2 * b] = q4.x; x.q[2 * b + 1] = q4.y; x.k[2 * b] = k4.x; x.k[2 * b + 1] = k4.y; x.a[2 * b] = a4.x; x.a[2 * b + 1] = a4.y;
                } else {
                    x.q[b] = *reinterpret_cast<const f2*>(qp);
                    x.k[b] = *reinterpret_cast<const f2*>(qp + TT * DP);
                    x.a[b] = *reinterpret_cast<const f2*>(qp + 2 * TT * DP);
                }
            }
            const ulonglong2 v4 = *reinterpret_cast<const ulonglong2*>(buf + 3 * TT * DP + 2 * (t * CB + wc));
            x.v[0] = v4.x; x.v[1] = v4.y;
        };
        auto token = [&](const Ops& x, float* o) {
            f2 na[RPL / 2];   // minus the rates
#pragma unroll
            for (int i = 0; i < RPL / 2; ++i) na[i] = x.a[i] ^ 0x8000000080000000ull;
#pragma unroll
            for (int c = 0; c < WALK_CW; ++c) {
                f2 acc = 0;   // (+0, +0)
#pragma unroll
                for (int i = 0; i < RPL / 2; ++i) {
                    s[c][i] = f2_fma(x.k[i], x.v[c], f2_fma(na[i], s[c][i], s[c][i]));
                    acc = f2_fma(s[c][i], x.q[i], acc);
                }
                float e, f;
                f2_unpack(acc, e, f);
                o[c] = e + f;
            }
        };
        auto leave = [&](const float* o, int t0) {
            const float sum = walk_sum<16>(o, lane);
            if (lane < 16) read[tile & 1][t0 + (mine >> 1)][wc + (mine & 1)] = sum;
        };
        if (qn - tile * TT >= TT) {
            float o[2 * TT];
            Ops x[2];
            load(x[0], 0);
#pragma unroll
            for (int t = 0; t < TT; ++t) {
                if (t + 1 < TT) load(x[(t + 1) & 1], t + 1);   // the next token's operands are on their way
                token(x[t & 1], o + 2 * t);
            }
            leave(o, 0);
            leave(o + TT, 8);
        } else {   // (a token that is not there leaves the state alone, whatever it holds)
#pragma unroll 1
            for (int t0 = 0; t0 < TT; t0 += 8) {
                float o[16];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    o[2 * u] = o[2 * u + 1] = 0.f;
                    if (tile * TT + t0 + u < qn) {
                        Ops x;
                        load(x, t0 + u);
                        token(x, o + 2 * u);
                    }
                }
                leave(o, t0);
            }
        }
    }
    __syncthreads();
    read_out(n_tiles - 1);
#pragma unroll
    for (int c = 0; c < WALK_CW; ++c)
#pragma unroll
        for (int i = 0; i < RPL / 2; ++i) {
            const int r = row_of(2 * i), col = col0 + wc + c;
            float e, f;
            f2_unpack(s[c][i], e, f);
            if (r < d && col < dv) S[static_cast<size_t>(r) * dv + col] = e;
            if (r + 1 < d && col < dv) S[static_cast<size_t>(r + 1) * dv + col] = f;
        }
}

// Few tokens a request.  128 threads: 16 columns x 8 groups of R consecutive rows (d <= 8 R).
template <int R>
__global__ void __launch_bounds__(128) gla_tokens_kernel(const GlaArgs a, int col_blocks) {
    constexpr int DP = 8 * R;
    __shared__ __align__(16) float ops[3][DP];
    __shared__ float part[4][16];
    pdl_entry();
    pdl_trigger();
    const int tid = threadIdx.x, rg = tid >> 4, c = tid & 15, wid = tid >> 5;
    const int seg = blockIdx.y, h = blockIdx.x / col_blocks, col = (blockIdx.x % col_blocks) * 16 + c;
    const int qn = a.seg_qn[seg], q0 = a.seg_q0[seg];
    if (qn <= 0) return;
    const int d = a.d, dv = a.dv;
    const bool col_ok = col < dv;
    float* S = a.state + static_cast<size_t>(a.state_slots[seg]) * a.slot_stride + static_cast<size_t>(h) * d * dv;
    float s[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int r = rg * R + i;
        s[i] = (r < d && col_ok) ? S[static_cast<size_t>(r) * dv + col] : 0.f;
    }
    for (int t = 0; t < qn; ++t) {
        const size_t row = static_cast<size_t>(q0 + t);
        const float vv = col_ok ? a.v[row * a.ldv + a.off_v + h * dv + col] : 0.f;
        for (int r = tid; r < DP; r += 128) {
            ops[0][r] = r < d ? a.q[row * a.ldq + a.off_q + h * d + r] : 0.f;
            ops[1][r] = r < d ? a.k[row * a.ldk + a.off_k + h * d + r] : 0.f;
            ops[2][r] = r < d ? a.a[row * a.lda + a.off_a + h * d + r] : 0.f;
        }
        __syncthreads();
        float o0 = 0.f, o1 = 0.f;
#pragma unroll
        for (int i = 0; i < R; i += 4) {
            const float4 qv = *reinterpret_cast<const float4*>(&ops[0][rg * R + i]);
            const float4 kv = *reinterpret_cast<const float4*>(&ops[1][rg * R + i]);
            const float4 av = *reinterpret_cast<const float4*>(&ops[2][rg * R + i]);
            s[i] = fmaf(kv.x, vv, fmaf(-av.x, s[i], s[i]));
            s[i + 1] = fmaf(kv.y, vv, fmaf(-av.y, s[i + 1], s[i + 1]));
            s[i + 2] = fmaf(kv.z, vv, fmaf(-av.z, s[i + 2], s[i + 2]));
            s[i + 3] = fmaf(kv.w, vv, fmaf(-av.w, s[i + 3], s[i + 3]));
            o0 = fmaf(s[i], qv.x, o0);
            o1 = fmaf(s[i + 1], qv.y, o1);
            o0 = fmaf(s[i + 2], qv.z, o0);
            o1 = fmaf(s[i + 3], qv.w, o1);
        }
        float o = o0 + o1;
        o += __shfl_xor_sync(0xffffffffu, o, 16);
        if ((tid & 31) < 16) part[wid][c] = o;
        __syncthreads();   // (also: nobody reads the operands any more)
        if (tid < 16 && col_ok)
            a.out[row * a.ldo + h * dv + col] = ((part[0][c] + part[1][c]) + (part[2][c] + part[3][c])) * a.q_scale;
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int r = rg * R + i;
        if (r < d && col_ok) S[static_cast<size_t>(r) * dv + col] = s[i];
    }
}

#define GC_D 128                 // channels of a head
#define GC_LD (GC_D + 8)         // bfloat16 from row to row of a chunk's operands (rows meet in no bank)
#define GC_ALD 24                // the same of a chunk's 16 x 16 matrices
#define GC_PART (CH * GC_LD)     // a part of q or k
#define GC_STAGE (2 * (6 * GC_PART + 3 * CH * GC_ALD) + 4 * GC_D)   // bytes: q, k, A, C
#define GC_STAGES 3

// What gla_chunk_prep leaves for rows w0 .. w1 of the step: a stage's bytes for every chunk and head, as they lie in shared memory.
struct GlaChunks {
    uint8_t* at;
    int w0, w1;
};
// A segment's rows within the window, and their chunks, which lie behind those of the segments before it in the list (whose rows may
// come in another order).  Every segment may leave one chunk unfilled.
__device__ __forceinline__ int gla_window(const GlaArgs& a, const GlaChunks& s, int seg, int& q0, int& qn) {
    const int first = a.seg_q0[seg], last = min(first + a.seg_qn[seg], s.w1);
    q0 = max(first, s.w0);
    qn = last - q0;
    return qn > 0 ? (qn + CH - 1) / CH : 0;
}
// The place of a segment's first chunk; a warp adds up.
__device__ __forceinline__ int gla_first_chunk(const GlaArgs& a, const GlaChunks& s, int seg) {
    int n = 0, q0, qn;
    for (int j = threadIdx.x & 31; j < seg; j += 32) n += gla_window(a, s, j, q0, qn);
    return __reduce_add_sync(0xffffffffu, n);
}
// The first row of the chunk in a place and the rows of its segment from there on (0: nobody's place); a warp looks.
__device__ __forceinline__ int gla_rows_at(const GlaArgs& a, const GlaChunks& s, int place, int n_seg, int& row0) {
    const int lane = threadIdx.x & 31;
    for (int j0 = 0; j0 < n_seg; j0 += 32) {
        int q0 = 0, qn = 0;
        const int n = j0 + lane < n_seg ? gla_window(a, s, j0 + lane, q0, qn) : 0;
        int upto = n;   // chunks of these 32 segments up to and with the lane's
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += x;
        }
        const unsigned behind = __ballot_sync(0xffffffffu, place < upto);
        if (behind) {
            const int t = (place - (upto - n)) * CH, from = __ffs(behind) - 1;
            row0 = __shfl_sync(0xffffffffu, q0 + t, from);
            return __shfl_sync(0xffffffffu, qn - t, from);
        }
        place -= __shfl_sync(0xffffffffu, upto, 31);
    }
    return 0;
}

// 64 threads to a chunk and head, two channels each; a block takes four heads of the chunk in place blockIdx.x.  The grid is of places, and every
// warp finds its place's segment (a grid of all rows times all segments has n_seg blocks for one that works, each of which counted
// through the list: 64 requests of 64 tokens, 16 heads 503 -> 295 us, of 4 heads 172 -> 63).
__global__ void __launch_bounds__(256) gla_chunk_prep(const GlaArgs a, const GlaChunks s, int n_seg) {
    __shared__ float sums[4][2][160];
    pdl_entry();
    pdl_trigger();
    int row0 = 0;
    const int live = min(CH, gla_rows_at(a, s, blockIdx.x, n_seg, row0));
    if (live <= 0) return;
    const int hl = threadIdx.x >> 6, h = blockIdx.y * 4 + hl, tid = threadIdx.x & 63, lane = tid & 31, half = tid >> 5;
    const bool on = h < a.H;
    const int d0 = 2 * tid, hh = on ? h : 0;
    float2 q[CH], k[CH], c[CH];
#pragma unroll
    for (int i = 0; i < CH; ++i) {
        q[i] = k[i] = c[i] = make_float2(0.f, 0.f);
        if (i < live) {
            const size_t row = static_cast<size_t>(row0 + i);
            q[i] = *reinterpret_cast<const float2*>(a.q + row * a.ldq + a.off_q + hh * GC_D + d0);
            k[i] = *reinterpret_cast<const float2*>(a.k + row * a.ldk + a.off_k + hh * GC_D + d0);
            c[i] = *reinterpret_cast<const float2*>(a.a + row * a.lda + a.off_a + hh * GC_D + d0);
        }
    }
    auto grow = [](float& x, float rate) { x += fmaf(-x, rate, rate); };   // 1 - (1 - x)(1 - rate)
    uint8_t* st = s.at + (static_cast<size_t>(blockIdx.x) * a.H + hh) * GC_STAGE;
    bf16* parts = reinterpret_cast<bf16*>(st);
    bf16* amat = parts + 6 * GC_PART;
    float* rates = reinterpret_cast<float*>(amat + 3 * CH * GC_ALD);
    auto leave = [&](int i, int which, float x, float y) {   // (rows that are not there: zeros)
        if (!on) return;
        uint32_t p[3];
        bf16_parts(x, y, p[0], p[1], p[2]);
#pragma unroll
        for (int j = 0; j < 3; ++j) *reinterpret_cast<uint32_t*>(parts + (3 * which + j) * GC_PART + i * GC_LD + d0) = p[j];
    };
    {
        float x = 0.f, y = 0.f;
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            grow(x, c[i].x);
            grow(y, c[i].y);
            leave(i, 0, fmaf(-x, q[i].x, q[i].x), fmaf(-y, q[i].y, q[i].y));
        }
        if (on) *reinterpret_cast<float2*>(rates + d0) = make_float2(x, y);
    }
    {
        float x = 0.f, y = 0.f;
#pragma unroll
        for (int j = CH - 1; j >= 0; --j) {
            leave(j, 1, fmaf(-x, k[j].x, k[j].x), fmaf(-y, k[j].y, k[j].y));
            grow(x, c[j].x);
            grow(y, c[j].y);
        }
    }
    // A: pair (j, i), i = j .. 15, is value 16 j - j (j - 1) / 2 + i - j; 32 values cross the lanes together
    float v[32];
    int n = 0;
#pragma unroll
    for (int j = 0; j < CH; ++j) {
        float x = k[j].x, y = k[j].y;
#pragma unroll
        for (int i = j; i < CH; ++i) {
            if (i > j) {
                x = fmaf(-x, c[i].x, x);
                y = fmaf(-y, c[i].y, y);
            }
            v[n & 31] = fmaf(q[i].x, x, q[i].y * y);
            if ((n & 31) == 31) sums[hl][half][(n & ~31) + walk_sum_index<32>(lane)] = walk_sum<32>(v, lane);
            ++n;
        }
    }
    {
        const float last = walk_sum<8>(v, lane);   // 136 = 4 x 32 + 8
        if (lane < 8) sums[hl][half][128 + walk_sum_index<8>(lane)] = last;
    }
    __syncthreads();
    if (!on) return;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int i = (tid + 64 * u) >> 3, j = 2 * (tid & 7);
        auto at = [&](int jj) -> float {
            const int x = 16 * jj - jj * (jj - 1) / 2 + i - jj;
            return jj <= i ? sums[hl][0][x] + sums[hl][1][x] : 0.f;
        };
        uint32_t p[3];
        bf16_parts(at(j), at(j + 1), p[0], p[1], p[2]);
#pragma unroll
        for (int m = 0; m < 3; ++m) *reinterpret_cast<uint32_t*>(amat + (m * CH + i) * GC_ALD + j) = p[m];
    }
}

// A block: sixteen columns of one head of one request; warp w keeps S^T of its sixteen columns x channels 16 w .. 16 w + 15, two
// tiles of sums (chunk_mma.cuh).  Two blocks an SM: 228 KB hold 3 stages and 25 KB of each.
__global__ void __launch_bounds__(256, 2) gla_chunk_kernel(const GlaArgs a, const GlaChunks s, int col_blocks) {
    extern __shared__ __align__(16) uint8_t gc_smem[];   // [GC_STAGES][GC_STAGE]
    __shared__ __align__(8) unsigned long long bars[GC_STAGES];
    __shared__ __align__(16) bf16 vt[2][3][CH][GC_ALD];  // v^T of a chunk: [parity][part][column][token]
    __shared__ float vf[3][CH][CH];                      // and as it is, copied two chunks ahead: [chunk][token][column]
    __shared__ float red[2][8][CH][CH + 4];              // read-outs of the warps: [parity][warp][token][column] (a warp's meet in no bank)
    pdl_entry();
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
    const int h = blockIdx.x / col_blocks, col0 = (blockIdx.x % col_blocks) * CH;
    int q0, qn;
    if (gla_window(a, s, blockIdx.y, q0, qn) == 0) return;
    const int chunk0 = gla_first_chunk(a, s, blockIdx.y);
    if (tid == 0) {
        for (int i = 0; i < GC_STAGES; ++i) ch_bar_init(ch_smem(&bars[i]));
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    const int dv = a.dv, n_chunks = (qn + CH - 1) / CH;
    float* S = a.state + static_cast<size_t>(a.state_slots[blockIdx.y]) * a.slot_stride + static_cast<size_t>(h) * GC_D * dv;
    const int vc = tid & 15, vtok = tid >> 4;   // this thread's value of v, and the read-out that it sums up

    auto fetch = [&](int c) {
        const int i = c % GC_STAGES;
        if (c < n_chunks)
            ch_bulk(ch_smem(gc_smem + i * GC_STAGE), s.at + (static_cast<size_t>(chunk0 + c) * a.H + h) * GC_STAGE, GC_STAGE, ch_smem(&bars[i]));
    };
    auto copy_v = [&](int c) {   // (a thread lays out what it copied itself)
        const int tok = c * CH + vtok;
        const bool live = tok < qn && col0 + vc < dv;
        walk_copy<4>(&vf[c % 3][vtok][vc], live ? a.v + static_cast<size_t>(q0 + tok) * a.ldv + a.off_v + h * dv + col0 + vc : a.v, live);
        walk_commit();
    };
    auto lay = [&](int c) -> bool {   // v into its places; false where it is not finite
        const float v = vf[c % 3][vtok][vc];
        uint32_t p[3];
        bf16_parts(v, 0.f, p[0], p[1], p[2]);
#pragma unroll
        for (int j = 0; j < 3; ++j) *reinterpret_cast<unsigned short*>(&vt[c & 1][j][vc][vtok]) = static_cast<unsigned short>(p[j]);
        return fabsf(v) < INFINITY;
    };
    if (tid == 0)
        for (int i = 0; i < GC_STAGES - 1; ++i) fetch(i);
    for (int c = 0; c < 2; ++c) copy_v(c);
    float sv[2][4];   // S^T: column g (+ 8 for the upper two), channel 16 w + 8 tile + 2 t (+ 1)
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int col = col0 + g + 8 * (e >> 1), d = 16 * w + 8 * n + 2 * t + (e & 1);
            sv[n][e] = col < dv ? S[static_cast<size_t>(d) * dv + col] : 0.f;
        }
    walk_wait<1>();
    bool plain = lay(0);   // this thread's value of the chunk is finite
    auto read_out = [&](int c, bool odd) {
        float sum = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) sum += red[c & 1][i][vtok][vc];
        if (odd) {   // a v that is not finite must not meet the zeros of A in front of it: what the MMAs left out
            const bf16* A = reinterpret_cast<const bf16*>(gc_smem + (c % GC_STAGES) * GC_STAGE) + 6 * GC_PART + vtok * GC_ALD;
            for (int j = 0; j <= vtok; ++j) {
                const float x = __bfloat162float(A[j]) + __bfloat162float(A[CH * GC_ALD + j]) + __bfloat162float(A[2 * CH * GC_ALD + j]);
                sum = fmaf(x, vf[c % 3][j][vc], sum);
            }
        }
        const int tok = c * CH + vtok;
        if (tok < qn && col0 + vc < dv) a.out[static_cast<size_t>(q0 + tok) * a.ldo + h * dv + col0 + vc] = sum * a.q_scale;
    };
    bool odd_before = false;
    for (int c = 0; c < n_chunks; ++c) {
        const bool odd = __syncthreads_or(!plain);   // the chunk before is left by all
        if (odd_before) {                            // (its A and v are read once more)
            read_out(c - 1, true);
            __syncthreads();
        }
        if (tid == 0) fetch(c + GC_STAGES - 1);
        ch_wait(ch_smem(&bars[c % GC_STAGES]), (c / GC_STAGES) & 1);
        const bf16* Q = reinterpret_cast<const bf16*>(gc_smem + (c % GC_STAGES) * GC_STAGE);
        const bf16* Kp = Q + 3 * GC_PART;
        const bf16* A = Q + 6 * GC_PART;
        const float* C = reinterpret_cast<const float*>(A + 3 * CH * GC_ALD);
        // the reading of S, o^T[column][token] over this warp's sixteen channels, and v^T k for its channels
        float o[2][4], u[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[n][e] = u[n][e] = 0.f;
        uint32_t sp[3][4], vp[3][4], bq[2][3][2], bk[2][3][2];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            uint32_t p[3];
            bf16_parts(sv[e >> 1][2 * (e & 1)], sv[e >> 1][2 * (e & 1) + 1], p[0], p[1], p[2]);
#pragma unroll
            for (int j = 0; j < 3; ++j) sp[j][e] = p[j];
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            ch_ldsm(vp[j], &vt[c & 1][j][(lane & 7) + 8 * ((lane >> 3) & 1)][8 * (lane >> 4)]);   // v^T: 16 columns x 16 tokens
            uint32_t r[4];
            ch_ldsm_t(r, Kp + j * GC_PART + (lane & 15) * GC_LD + 16 * w + 8 * (lane >> 4));
            bk[0][j][0] = r[0]; bk[0][j][1] = r[1]; bk[1][j][0] = r[2]; bk[1][j][1] = r[3];
            ch_ldsm(r, Q + j * GC_PART + ((lane & 7) + 8 * (lane >> 4)) * GC_LD + 16 * w + 8 * ((lane >> 3) & 1));
            bq[0][j][0] = r[0]; bq[0][j][1] = r[1]; bq[1][j][0] = r[2]; bq[1][j][1] = r[3];
        }
        // (the four sums' products in turn)
#define GC_STEP(P) ch_mma_part<P>(u[0], vp, bk[0]); ch_mma_part<P>(o[0], sp, bq[0]); ch_mma_part<P>(u[1], vp, bk[1]); ch_mma_part<P>(o[1], sp, bq[1]);
        GC_STEP(0) GC_STEP(1) GC_STEP(2) GC_STEP(3) GC_STEP(4) GC_STEP(5)
#undef GC_STEP
        if (!odd && w == (c & 7)) {   // the chunk's own tokens: one warp's share, in turn
            uint32_t ba[2][3][2];
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                uint32_t r[4];
                ch_ldsm(r, A + (j * CH + (lane & 7) + 8 * (lane >> 4)) * GC_ALD + 8 * ((lane >> 3) & 1));
                ba[0][j][0] = r[0]; ba[0][j][1] = r[1]; ba[1][j][0] = r[2]; ba[1][j][1] = r[3];
            }
            ch_mma_pair(o, vp, ba);
        }
        // while the MMAs run: the chunk before is summed up, the next one's v laid out
        if (c > 0 && !odd_before) read_out(c - 1, false);
        copy_v(c + 2);
        walk_wait<1>();
        if (c + 1 < n_chunks) plain = lay(c + 1);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const float2 rate = *reinterpret_cast<const float2*>(C + 16 * w + 8 * n + 2 * t);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                red[c & 1][w][8 * n + 2 * t + (e & 1)][g + 8 * (e >> 1)] = o[n][e];
                sv[n][e] = fmaf(-((e & 1) ? rate.y : rate.x), sv[n][e], sv[n][e]) + u[n][e];   // S <- S - C S + v^T k
            }
        }
        odd_before = odd;
    }
    walk_wait<0>();
    __syncthreads();
    read_out(n_chunks - 1, odd_before);
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int col = col0 + g + 8 * (e >> 1), d = 16 * w + 8 * n + 2 * t + (e & 1);
            if (col < dv) S[static_cast<size_t>(d) * dv + col] = sv[n][e];
        }
}

// Rows of a step whose chunks scratch of `bytes` holds, with one unfilled chunk a segment; in whole chunks.
static long long gla_chunk_rows(int H, int n_seg, long long bytes) {
    const long long chunks = bytes / (static_cast<long long>(H) * GC_STAGE) - n_seg;
    return chunks > 0 ? chunks * CH : 0;
}

static int gla_chunks(const GlaArgs& a, int n_seg, int n_rows, void* scratch, long long scratch_bytes, cudaStream_t stream) {
    const long long rows = gla_chunk_rows(a.H, n_seg, scratch_bytes);
    const cudaError_t e = cudaFuncSetAttribute(gla_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GC_STAGES * GC_STAGE);
    if (e != cudaSuccess) return static_cast<int>(e);
    const int col_blocks = ceil_div(a.dv, CH);
    for (long long w0 = 0; w0 < n_rows; w0 += rows) {
        GlaChunks s;
        s.w0 = static_cast<int>(w0);
        s.w1 = static_cast<int>(w0 + rows < n_rows ? w0 + rows : n_rows);
        s.at = static_cast<uint8_t*>(scratch);
        locus_launch(gla_chunk_prep, dim3(ceil_div(s.w1 - s.w0, CH) + n_seg, ceil_div(a.H, 4)), dim3(256), 0, stream, a, s, n_seg);
        locus_launch(gla_chunk_kernel, dim3(a.H * col_blocks, n_seg), dim3(256), GC_STAGES * GC_STAGE, stream, a, s, col_blocks);
    }
    return locus_launch_status();
}

// Reads and clears the module's error word (0 = no bounded wait ran out).  Synchronises.
extern "C" int locus_gla_error() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_chunk_error, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) cudaMemcpyToSymbol(g_chunk_error, &zero, sizeof(int));
    return v;
}

// z [T, ld] float32, columns [off, off + n): z <- 1 - exp(-softplus(-z) / tau).
__global__ void __launch_bounds__(256) gla_decay_kernel(float* __restrict__ z, int ld, int off, int n, float inv_tau,
                                                        long long total) {
    pdl_entry();
    pdl_trigger();
    const long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
    if (i >= total) return;
    float* p = z + (i / n) * ld + off + (i % n);
    const float x = -*p;                                          // softplus(x) = max(x, 0) + log1p(exp(-|x|))
    const float sp = fmaxf(x, 0.f) + log1pf(expf(-fabsf(x)));
    *p = -expm1f(-sp * inv_tau);
}

extern "C" int locus_gla_decay(float* z, int ld, int off, int n, int T, float tau, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (n <= 0 || off < 0 || ld < off + n || !(tau > 0.f)) return LOCUS_ERR_UNSUPPORTED;
    const long long total = static_cast<long long>(T) * n;
    const long long blocks = (total + 255) / 256;
    if (blocks > 0x7fffffffLL) return LOCUS_ERR_UNSUPPORTED;
    locus_launch(gla_decay_kernel, dim3(static_cast<unsigned>(blocks)), dim3(256), 0, stream, z, ld, off, n, 1.0f / tau, total);
    return locus_launch_status();
}

template <int RPL, bool MIXED>
static int gla_walk(const GlaArgs& a, bool vec, int n_seg, cudaStream_t stream) {
    constexpr int CB = WALK_CW * WALK_WARPS;
    constexpr size_t smem = sizeof(float) * GL_STAGES * GL_TT * (3 * 32 * RPL + 2 * CB);
    const int col_blocks = (a.dv + CB - 1) / CB;
    auto* kernel = vec ? gla_walk_kernel<RPL, true, MIXED> : gla_walk_kernel<RPL, false, MIXED>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    locus_launch(kernel, dim3(a.H * col_blocks, n_seg), dim3(32 * WALK_WARPS), smem, stream, a, col_blocks,
                 walk_few(static_cast<long long>(a.H) * col_blocks * n_seg));
    return locus_launch_status();
}

// n_rows: the rows of `out`, which bound the tokens of all segments together.  At most two a segment (decoding), or no
// more than a lone request of few tokens: the tokens kernel.  Where portions may stand beside single tokens each block of the walk
// looks at its own request: a prompt portion of 100 tokens beside 32 decoding requests, 16 heads of 128, takes 30 us;
// all of it in tiles took 96, all of it token by token 52.
extern "C" int locus_gla_scan(const float* q, int ldq, int off_q, const float* k, int ldk, int off_k, const float* v, int ldv,
                              int off_v, const float* dec, int lda, int off_a, float* state, long long slot_stride,
                              const int* state_slots, const int* seg_q0, const int* seg_qn, int n_seg, int n_rows, float* out,
                              int ldo, int H, int d, int dv, float q_scale, void* scratch, long long scratch_bytes,
                              cudaStream_t stream) {
    if (n_seg <= 0) return 0;
    if (H <= 0 || d <= 0 || d > 256 || dv <= 0 || n_seg > 65535 || H > 65535) return LOCUS_ERR_UNSUPPORTED;
    GlaArgs a;
    a.q = q; a.k = k; a.v = v; a.a = dec; a.state = state; a.state_slots = state_slots; a.seg_q0 = seg_q0; a.seg_qn = seg_qn;
    a.out = out; a.slot_stride = slot_stride; a.ldq = ldq; a.off_q = off_q; a.ldk = ldk; a.off_k = off_k; a.ldv = ldv;
    a.off_v = off_v; a.lda = lda; a.off_a = off_a; a.ldo = ldo; a.H = H; a.d = d; a.dv = dv; a.q_scale = q_scale;
    if (walk_not_needed(n_rows, n_seg, d)) {
        const int col_blocks = (dv + 15) / 16;
        const dim3 grid(H * col_blocks, n_seg);
        if (d <= 32) locus_launch(gla_tokens_kernel<4>, grid, dim3(128), 0, stream, a, col_blocks);
        else if (d <= 64) locus_launch(gla_tokens_kernel<8>, grid, dim3(128), 0, stream, a, col_blocks);
        else if (d <= 128) locus_launch(gla_tokens_kernel<16>, grid, dim3(128), 0, stream, a, col_blocks);
        else locus_launch(gla_tokens_kernel<32>, grid, dim3(128), 0, stream, a, col_blocks);
        return locus_launch_status();
    }
    const bool mixed = walk_may_be_mixed(n_rows, n_seg);
    const bool vec = ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(dec)) & 15) == 0 &&
                     ((ldq | off_q | ldk | off_k | lda | off_a | d) & 3) == 0;
    if (scratch != nullptr && vec && d == GC_D && (reinterpret_cast<uintptr_t>(scratch) & 15) == 0 && gla_chunk_rows(H, n_seg, scratch_bytes) > 0)
        return gla_chunks(a, n_seg, n_rows, scratch, scratch_bytes, stream);
    if (d <= 64) return mixed ? gla_walk<2, true>(a, vec, n_seg, stream) : gla_walk<2, false>(a, vec, n_seg, stream);
    if (d <= 128) return mixed ? gla_walk<4, true>(a, vec, n_seg, stream) : gla_walk<4, false>(a, vec, n_seg, stream);
    return mixed ? gla_walk<8, true>(a, vec, n_seg, stream) : gla_walk<8, false>(a, vec, n_seg, stream);
}
