// The gated delta rule: per request and head a matrix state S [d, dv] (float32, in the request's state slot, zero
// when the request opens) that every token first decays, then corrects towards its value along its key, then reads:
//
//     S <- g_t S;     u_t = beta_t (v_t - S^T k_t);     S <- S + k_t u_t^T;     o_t = S^T q_t,
//
// with g_t (a decay in (0, 1]) and beta_t (a step in (0, 1)) one float32 number per token and head, made by the
// caller.  q and k of head h are those of its group h / heads_per_group; v is the head's own.  Everything is float32;
// q, k and v are columns of float32 row matrices given by pointer, row stride and offset.
//
// The columns of S do not meet: with a = S_old^T k, b = S_old^T q (both of the state BEFORE the token) and the number
// k . q, u = beta (v - g a) and o = g b + u (k . q).  So a token costs one round of sums across lanes, not two in a row.
//
//   delta_walk   for portions.  A block of eight warps owns 16 columns of one head's state for one request and walks the
//                request's new tokens four at a time, the state in registers (walk.cuh says which lane holds what).  The
//                sums a_t and b_t of four tokens are all taken against the state in front of the four, so that they cross
//                the row groups together, once, and what a token's write adds to the later ones is a number per pair of
//                tokens: with G_t = g_0 .. g_t within the four,
//                    u_t = beta_t v_t - beta_t G_t a_t - beta_t sum_(j < t) (g_(j+1) .. g_t) (k_j . k_t) u_j
//                    o_t = G_t b_t + sum_(j <= t) (g_(j+1) .. g_t) (k_j . q_t) u_j
//                    S  <- G_3 S + sum_j (g_(j+1) .. g_3) k_j u_j^T
//                (products of decays only, nothing is divided).  The pairs' numbers are formed once per block for 16
//                tokens, two threads to a pair; q, k, v, beta and the decays of 16 tokens are copied into shared memory
//                together, asynchronously, two tiles ahead.  One token at a time with a warp's own fetch one token ahead,
//                a token took 385 ns (one request of 2,048 tokens, 16 heads of 128 x 128: 788 us, eight such requests 4,470 us): a
//                chain of fetch, sums, three exchanges and update that the next token waited for.  Now 440 and 2,030 us, three
//                requests of 700 tokens 308.  (Eight tokens together: 454, 2,400 and 379 us: fewer crossings, but two
//                blocks an SM instead of three.)
//   delta_tokens for steps of few tokens a request (decoding): 16 columns of a head and 8 groups of rows to a block, so that
//                a row of the state is read and written in whole sectors (64 requests: 51 -> 28 us).
//   delta_out    a head's read-out divided by its root mean square, times a weight, times silu(gate).
#include "common.cuh"
#include "walk.cuh"

struct DeltaArgs {
    const float* q;
    const float* k;
    const float* v;
    const float* beta;    // [T, H]
    const float* decay;   // [T, H]
    float* state;
    const int* state_slots;
    const int* seg_q0;
    const int* seg_qn;
    float* out;           // [T, ldo]: head h's columns start at h * dv
    long long slot_stride;
    int ldq, off_q, ldk, off_k, ldv, off_v, ldo;
    int H, heads_per_group, d, dv;
};

// A request of few tokens in a walk's block of 256 threads: 32 columns from col0 on x 8 groups of R consecutive rows (d <= 8 R), the
// sums of a column as delta_tokens_kernel below takes them (which as an instance of this function ran 7 to 11 % longer).
// part: [3][4][16] for either half of the columns.
template <int R>
__device__ __forceinline__ void delta_few(const DeltaArgs& a, int seg, int h, int col0, float (*ops)[8 * R], float (*part)[4][16]) {
    constexpr int DP = 8 * R;
    const int tid = threadIdx.x, half = tid >> 7, rg = (tid & 127) >> 4, c = tid & 15, wid = (tid & 127) >> 5;
    const int col = col0 + 16 * half + c;
    const int qn = a.seg_qn[seg], q0 = a.seg_q0[seg];
    const int d = a.d, dv = a.dv, g = h / a.heads_per_group;
    part += 3 * half;
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
        const float beta = a.beta[row * a.H + h], gd = a.decay[row * a.H + h];
        for (int r = tid; r < DP; r += 256) {
            ops[0][r] = r < d ? a.q[row * a.ldq + a.off_q + g * d + r] : 0.f;
            ops[1][r] = r < d ? a.k[row * a.ldk + a.off_k + g * d + r] : 0.f;
        }
        __syncthreads();
        float sk0 = 0.f, sk1 = 0.f, sq0 = 0.f, sq1 = 0.f, kq0 = 0.f, kq1 = 0.f;
#pragma unroll
        for (int i = 0; i < R; i += 2) {
            const float2 qv = *reinterpret_cast<const float2*>(&ops[0][rg * R + i]);
            const float2 kv = *reinterpret_cast<const float2*>(&ops[1][rg * R + i]);
            sk0 = fmaf(s[i], kv.x, sk0);
            sq0 = fmaf(s[i], qv.x, sq0);
            kq0 = fmaf(kv.x, qv.x, kq0);
            sk1 = fmaf(s[i + 1], kv.y, sk1);
            sq1 = fmaf(s[i + 1], qv.y, sq1);
            kq1 = fmaf(kv.y, qv.y, kq1);
        }
        float sk = sk0 + sk1, sq = sq0 + sq1, kq = kq0 + kq1;
        sk += __shfl_xor_sync(0xffffffffu, sk, 16);
        sq += __shfl_xor_sync(0xffffffffu, sq, 16);
        kq += __shfl_xor_sync(0xffffffffu, kq, 16);
        if ((tid & 31) < 16) {
            part[0][wid][c] = sk;
            part[1][wid][c] = sq;
            part[2][wid][c] = kq;
        }
        __syncthreads();
        sk = (part[0][0][c] + part[0][1][c]) + (part[0][2][c] + part[0][3][c]);
        sq = (part[1][0][c] + part[1][1][c]) + (part[1][2][c] + part[1][3][c]);
        kq = (part[2][0][c] + part[2][1][c]) + (part[2][2][c] + part[2][3][c]);
        const float u = beta * (vv - gd * sk);
#pragma unroll
        for (int i = 0; i < R; i += 2) {
            const float2 kv = *reinterpret_cast<const float2*>(&ops[1][rg * R + i]);
            s[i] = fmaf(gd, s[i], kv.x * u);
            s[i + 1] = fmaf(gd, s[i + 1], kv.y * u);
        }
        if (rg == 0 && col_ok) a.out[row * a.ldo + h * dv + col] = fmaf(u, kq, gd * sq);
        if (t + 1 < qn) __syncthreads();   // nobody reads this token's operands and sums any more
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int r = rg * R + i;
        if (r < d && col_ok) S[static_cast<size_t>(r) * dv + col] = s[i];
    }
}

#define DR_STAGES 3
#define DR_TT 16       // tokens of a tile
#define DR_G 4         // tokens that are worked on together
// numbers of four tokens: beta G, G, E, beta (4 each); then rows 1 .. 3 of L, then rows 0 .. 3 of P (4 each, of row t the first t + 1)
#define DR_L (4 * DR_G)
#define DR_P (DR_L + DR_G * (DR_G - 1))
#define DR_COEF (DR_P + DR_G * DR_G)

// RPL: rows of a column that a lane keeps, of two columns (d <= 32 RPL).  VEC: q's and k's rows of a head start on 16-byte
// boundaries and d is a multiple of 4, so four rows are one copy.  MIXED: requests of up to `few` tokens are taken token by token.
template <int RPL, bool VEC, bool MIXED>
__global__ void __launch_bounds__(32 * WALK_WARPS, RPL > 4 ? 2 : 3) delta_walk_kernel(const DeltaArgs a, int col_blocks, int few) {
    constexpr int DP = 32 * RPL, LD = DP + 8, TT = DR_TT, CB = WALK_CW * WALK_WARPS, NT = 32 * WALK_WARPS;
    constexpr int RV = RPL < 4 ? RPL : 4;          // rows of a load
    constexpr int TILE = TT * (2 * LD + CB + 2);   // q, k: [TT][LD]; v: [TT][CB]; beta, decay: [TT]
    extern __shared__ __align__(16) float walk_smem[];   // [DR_STAGES][TILE], then [TT / DR_G][DR_COEF]
    __shared__ __align__(16) f2 writes[WALK_WARPS][DR_G][WALK_CW];   // a warp's u of four tokens, each twice
    float* coef = walk_smem + DR_STAGES * TILE;
    pdl_entry();
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int seg = blockIdx.y, h = blockIdx.x / col_blocks, col0 = (blockIdx.x % col_blocks) * CB;
    const int qn = a.seg_qn[seg], q0 = a.seg_q0[seg];
    if (qn <= 0) return;
    static_assert(NT == 256 && CB == 16, "delta_few takes the columns of two blocks");
    if (MIXED && qn <= few) {   // a request of few tokens beside portions: every other block does two blocks' columns
        if ((blockIdx.x % col_blocks) & 1) return;
        float (*part)[4][16] = reinterpret_cast<float (*)[4][16]>(walk_smem + 2 * DP);
        if (RPL == 2 && a.d <= 32) delta_few<4>(a, seg, h, col0, reinterpret_cast<float (*)[32]>(walk_smem), part);
        else delta_few<4 * RPL>(a, seg, h, col0, reinterpret_cast<float (*)[DP]>(walk_smem), part);
        return;
    }
    const int d = a.d, dv = a.dv, wc = wid * WALK_CW, col = col0 + wc;
    float* S = a.state + static_cast<size_t>(a.state_slots[seg]) * a.slot_stride + static_cast<size_t>(h) * d * dv;
    const int g = h / a.heads_per_group;

    // rows d .. DP of the tiles are never copied: they stay zero, and so do the state's rows there
    if (d < DP)
        for (int i = tid; i < DR_STAGES * TT * 2 * (DP - d); i += NT) {
            const int row = i / (DP - d), r = d + i % (DP - d);
            walk_smem[(row / (2 * TT)) * TILE + (row % (2 * TT)) * LD + r] = 0.f;
        }
    const float* src[2] = {a.q + a.off_q + g * d, a.k + a.off_k + g * d};
    const int ld[2] = {a.ldq, a.ldk};
    const float* vsrc = a.v + a.off_v + h * dv + col0;
    auto fetch = [&](int tile) {   // a tile's operands into its buffer; tokens behind the last one are zeros
        float* buf = walk_smem + (tile % DR_STAGES) * TILE;
#pragma unroll
        for (int w = 0; w < 2; ++w)
#pragma unroll
            for (int i = 0; i < TT / WALK_WARPS; ++i) {
                const int t = wid + i * WALK_WARPS, tok = tile * TT + t;
                const bool live = tok < qn;
                const float* row = src[w] + static_cast<size_t>(q0 + (live ? tok : 0)) * ld[w];
                float* dst = buf + (w * TT + t) * LD;
                if (VEC) {
                    for (int r = 4 * lane; r < d; r += 128) walk_copy<16>(dst + r, row + r, live);
                } else {
                    for (int r = lane; r < d; r += 32) walk_copy<4>(dst + r, row + r, live);
                }
            }
        static_assert(TT * CB == NT, "a value of a tile to a thread");
        {
            const int t = tid / CB, c = tid % CB, tok = tile * TT + t;
            const bool live = tok < qn && col0 + c < dv;
            walk_copy<4>(buf + 2 * TT * LD + tid, vsrc + (live ? static_cast<size_t>(q0 + tok) * a.ldv + c : 0), live);
        }
        if (tid < 2 * TT) {
            const int t = tid % TT, tok = tile * TT + t;
            const bool live = tok < qn;
            walk_copy<4>(buf + TT * (2 * LD + CB) + tid,
                         (tid < TT ? a.beta : a.decay) + static_cast<size_t>(q0 + (live ? tok : 0)) * a.H + h, live);
        }
    };
    const int n_tiles = (qn + TT - 1) / TT;
#pragma unroll
    for (int i = 0; i < DR_STAGES - 1; ++i) {
        if (i < n_tiles) fetch(i);
        walk_commit();
    }
    auto row_of = [&](int i) { return 128 * (i / RV) + RV * lane + (i % RV); };
    f2 s[2][RPL / 2];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < RPL / 2; ++i) {
            const int r = row_of(2 * i);
            s[j][i] = f2_pack((r < d && col + j < dv) ? S[static_cast<size_t>(r) * dv + col + j] : 0.f,
                              (r + 1 < d && col + j < dv) ? S[static_cast<size_t>(r + 1) * dv + col + j] : 0.f);
        }
    // The pair of tokens j <= t of the four that this thread's half of a sum belongs to: of the 16 pairs of a group, 6
    // k_j . k_t (j < t) and 10 k_j . q_t; a pair is (row, column): j and t of k_j . q_t where row <= column, and elsewhere t
    // and j of k_j . k_t.
    constexpr int PAIRS = DR_G * DR_G;
    const int half = tid & 1, pair = (tid >> 1) % PAIRS, group = tid / (2 * PAIRS);
    const int pr = pair % DR_G, pc = pair / DR_G;
    const bool with_q = pr <= pc;
    const int pj = with_q ? pr : pc, pt = with_q ? pc : pr;
    // of the 16 sums (a or b, token, column) of four tokens, the one that this lane ends up with
    const int mine = walk_sum_index<4 * DR_G>(lane), my_t = (mine >> 1) % DR_G, my_c = mine & 1;
    const bool my_b = mine >= 2 * DR_G;
    for (int tile = 0; tile < n_tiles; ++tile) {
        walk_wait<DR_STAGES - 2>();
        __syncthreads();   // the tile is there for all warps, and nobody reads the buffer and the numbers that are written next
        if (tile + DR_STAGES - 1 < n_tiles) fetch(tile + DR_STAGES - 1);
        walk_commit();
        const float* qs = walk_smem + (tile % DR_STAGES) * TILE;
        const float* ks = qs + TT * LD;
        const float* vs = ks + TT * LD;
        const float* bs = vs + TT * CB;
        if (group < TT / DR_G) {   // (rows LD = DP + 8 floats apart and the halves of a sum four floats apart meet in no bank)
            const float* x = ks + (DR_G * group + pj) * LD + 4 * half;
            const float* y = (with_q ? qs : ks) + (DR_G * group + pt) * LD + 4 * half;
            float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;
#pragma unroll
            for (int i = 0; i < DP / 8; ++i) {
                const float4 xv = *reinterpret_cast<const float4*>(x + 8 * i), yv = *reinterpret_cast<const float4*>(y + 8 * i);
                d0 = fmaf(xv.x, yv.x, d0);
                d1 = fmaf(xv.y, yv.y, d1);
                d2 = fmaf(xv.z, yv.z, d2);
                d3 = fmaf(xv.w, yv.w, d3);
            }
            float dot = (d0 + d1) + (d2 + d3);
            dot += __shfl_xor_sync(0xffffffffu, dot, 1);
            float w = 1.f, before = 1.f, behind = 1.f;   // g_(j+1) .. g_t; g_0 .. g_t; g_(t+1) .. g_3
#pragma unroll
            for (int i = 0; i < DR_G; ++i) {
                const float gi = tile * TT + DR_G * group + i < qn ? bs[TT + DR_G * group + i] : 1.f;
                if (i > pj && i <= pt) w *= gi;
                if (i <= pt) before *= gi;
                if (i > pt) behind *= gi;
            }
            const float beta = bs[DR_G * group + pt];
            float* c = coef + group * DR_COEF;
            if (half == 0) {
                if (with_q) c[DR_P + DR_G * pt + pj] = w * dot;
                else c[DR_L + DR_G * (pt - 1) + pj] = -beta * w * dot;
            } else if (pj == pt) {
                c[pt] = beta * before;
                c[DR_G + pt] = before;
                c[2 * DR_G + pt] = behind;
                c[3 * DR_G + pt] = beta;
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int t0 = 0; t0 < TT && tile * TT + t0 < qn; t0 += DR_G) {
            const float* c = coef + (t0 / DR_G) * DR_COEF;
            const int live = qn - tile * TT - t0;
            f2 kk[DR_G][RPL / 2];
            float sums[4 * DR_G];
#pragma unroll
            for (int t = 0; t < DR_G; ++t) {
                f2 qv[RPL / 2];
                const float* kp = ks + (t0 + t) * LD + RV * lane;
                const float* qp = qs + (t0 + t) * LD + RV * lane;
#pragma unroll
                for (int b = 0; b < RPL / RV; ++b) {
                    if constexpr (RV == 4) {
                        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(kp + 128 * b);
                        const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(qp + 128 * b);
                        kk[t][2 * b] = x.x; kk[t][2 * b + 1] = x.y; qv[2 * b] = y.x; qv[2 * b + 1] = y.y;
                    } else {
                        kk[t][b] = *reinterpret_cast<const f2*>(kp);
                        qv[b] = *reinterpret_cast<const f2*>(qp);
                    }
                }
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    f2 ka = 0, qa = 0;
#pragma unroll
                    for (int i = 0; i < RPL / 2; ++i) {
                        ka = f2_fma(s[j][i], kk[t][i], ka);
                        qa = f2_fma(s[j][i], qv[i], qa);
                    }
                    float e, f;
                    f2_unpack(ka, e, f);
                    sums[2 * t + j] = e + f;
                    f2_unpack(qa, e, f);
                    sums[2 * DR_G + 2 * t + j] = e + f;
                }
            }
            const float sum = walk_sum<4 * DR_G>(sums, lane);
            // u of the four tokens, of this lane's column, by every lane: a of token t comes from the lane that ended up with it
            auto four = [&](int at) { return *reinterpret_cast<const float4*>(c + at); };
            float u[DR_G];
            const float* vp = vs + t0 * CB + wc + my_c;
#pragma unroll
            for (int t = 0; t < DR_G; t += 4) {
                const float4 bG = four(t), be = four(3 * DR_G + t);
                auto a_of = [&](int i) { return __shfl_sync(0xffffffffu, sum, walk_sum_index<4 * DR_G>(2 * (t + i) + my_c)); };
                u[t] = fmaf(-bG.x, a_of(0), be.x * vp[t * CB]);
                u[t + 1] = fmaf(-bG.y, a_of(1), be.y * vp[(t + 1) * CB]);
                u[t + 2] = fmaf(-bG.z, a_of(2), be.z * vp[(t + 2) * CB]);
                u[t + 3] = fmaf(-bG.w, a_of(3), be.w * vp[(t + 3) * CB]);
            }
            float p[DR_G];
#pragma unroll
            for (int t = 0; t < DR_G; t += 4) *reinterpret_cast<float4*>(p + t) = four(DR_P + DR_G * my_t + t);
            float o = c[DR_G + my_t] * sum;
#pragma unroll
            for (int t = 0; t < DR_G; ++t) {
                if (t > 0) {
                    float l[DR_G];
#pragma unroll
                    for (int j = 0; j < t; j += 4) *reinterpret_cast<float4*>(l + j) = four(DR_L + DR_G * (t - 1) + j);
#pragma unroll
                    for (int j = 0; j < t; ++j) u[t] = fmaf(l[j], u[j], u[t]);
                }
                if (t >= live) u[t] = 0.f;   // (a token that is not there writes nothing, whatever the state holds)
                if (t <= my_t) o = fmaf(p[t], u[t], o);   // (not 0 * u behind it: a u that is not finite stays with its token and later ones)
            }
            if (my_b) {
                const int tok = tile * TT + t0 + my_t;
                if (tok < qn && col + my_c < dv) a.out[static_cast<size_t>(q0 + tok) * a.ldo + h * dv + col + my_c] = o;
            } else {
                float w = u[0];
#pragma unroll
                for (int t = 1; t < DR_G; ++t) w = my_t == t ? u[t] : w;
                w *= c[2 * DR_G + my_t];
                writes[wid][my_t][my_c] = f2_pack(w, w);
            }
            __syncwarp();
            const float G = c[2 * DR_G - 1];
            const f2 G2 = f2_pack(G, G);
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int i = 0; i < RPL / 2; ++i) s[j][i] = f2_mul(G2, s[j][i]);
#pragma unroll
            for (int t = 0; t < DR_G; ++t) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(&writes[wid][t][0]);
#pragma unroll
                for (int i = 0; i < RPL / 2; ++i) {
                    s[0][i] = f2_fma(kk[t][i], w.x, s[0][i]);
                    s[1][i] = f2_fma(kk[t][i], w.y, s[1][i]);
                }
            }
            __syncwarp();   // nobody reads the writes any more
        }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < RPL / 2; ++i) {
            const int r = row_of(2 * i);
            float e, f;
            f2_unpack(s[j][i], e, f);
            if (r < d && col + j < dv) S[static_cast<size_t>(r) * dv + col + j] = e;
            if (r + 1 < d && col + j < dv) S[static_cast<size_t>(r + 1) * dv + col + j] = f;
        }
}

// Few tokens a request.  128 threads: 16 columns x 8 groups of R consecutive rows (d <= 8 R).
template <int R>
__global__ void __launch_bounds__(128) delta_tokens_kernel(const DeltaArgs a, int col_blocks) {
    constexpr int DP = 8 * R;
    __shared__ __align__(16) float ops[2][DP];
    __shared__ float part[3][4][16];
    pdl_entry();
    pdl_trigger();
    const int tid = threadIdx.x, rg = tid >> 4, c = tid & 15, wid = tid >> 5;
    const int seg = blockIdx.y, h = blockIdx.x / col_blocks, col = (blockIdx.x % col_blocks) * 16 + c;
    const int qn = a.seg_qn[seg], q0 = a.seg_q0[seg];
    if (qn <= 0) return;
    const int d = a.d, dv = a.dv, g = h / a.heads_per_group;
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
        const float beta = a.beta[row * a.H + h], gd = a.decay[row * a.H + h];
        for (int r = tid; r < DP; r += 128) {
            ops[0][r] = r < d ? a.q[row * a.ldq + a.off_q + g * d + r] : 0.f;
            ops[1][r] = r < d ? a.k[row * a.ldk + a.off_k + g * d + r] : 0.f;
        }
        __syncthreads();
        float sk0 = 0.f, sk1 = 0.f, sq0 = 0.f, sq1 = 0.f, kq0 = 0.f, kq1 = 0.f;
#pragma unroll
        for (int i = 0; i < R; i += 2) {
            const float2 qv = *reinterpret_cast<const float2*>(&ops[0][rg * R + i]);
            const float2 kv = *reinterpret_cast<const float2*>(&ops[1][rg * R + i]);
            sk0 = fmaf(s[i], kv.x, sk0);
            sq0 = fmaf(s[i], qv.x, sq0);
            kq0 = fmaf(kv.x, qv.x, kq0);
            sk1 = fmaf(s[i + 1], kv.y, sk1);
            sq1 = fmaf(s[i + 1], qv.y, sq1);
            kq1 = fmaf(kv.y, qv.y, kq1);
        }
        float sk = sk0 + sk1, sq = sq0 + sq1, kq = kq0 + kq1;
        sk += __shfl_xor_sync(0xffffffffu, sk, 16);
        sq += __shfl_xor_sync(0xffffffffu, sq, 16);
        kq += __shfl_xor_sync(0xffffffffu, kq, 16);
        if ((tid & 31) < 16) {
            part[0][wid][c] = sk;
            part[1][wid][c] = sq;
            part[2][wid][c] = kq;
        }
        __syncthreads();
        sk = (part[0][0][c] + part[0][1][c]) + (part[0][2][c] + part[0][3][c]);
        sq = (part[1][0][c] + part[1][1][c]) + (part[1][2][c] + part[1][3][c]);
        kq = (part[2][0][c] + part[2][1][c]) + (part[2][2][c] + part[2][3][c]);
        const float u = beta * (vv - gd * sk);
#pragma unroll
        for (int i = 0; i < R; i += 2) {
            const float2 kv = *reinterpret_cast<const float2*>(&ops[1][rg * R + i]);
            s[i] = fmaf(gd, s[i], kv.x * u);
            s[i + 1] = fmaf(gd, s[i + 1], kv.y * u);
        }
        if (rg == 0 && col_ok) a.out[row * a.ldo + h * dv + col] = fmaf(u, kq, gd * sq);
        if (t + 1 < qn) __syncthreads();   // nobody reads this token's operands and sums any more
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int r = rg * R + i;
        if (r < d && col_ok) S[static_cast<size_t>(r) * dv + col] = s[i];
    }
}

template <int RPL, bool MIXED>
static int delta_walk(const DeltaArgs& a, bool vec, int n_seg, cudaStream_t stream) {
    constexpr int CB = WALK_CW * WALK_WARPS;
    constexpr size_t smem = sizeof(float) * (DR_STAGES * DR_TT * (2 * (32 * RPL + 8) + CB + 2) + DR_TT / DR_G * DR_COEF);
    static_assert(DR_TT / DR_G * 2 * DR_G * DR_G <= 32 * WALK_WARPS, "two threads to a pair of tokens");
    const int col_blocks = (a.dv + CB - 1) / CB;
    auto* kernel = vec ? delta_walk_kernel<RPL, true, MIXED> : delta_walk_kernel<RPL, false, MIXED>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    locus_launch(kernel, dim3(a.H * col_blocks, n_seg), dim3(32 * WALK_WARPS), smem, stream, a, col_blocks,
                 walk_few(static_cast<long long>(a.H) * col_blocks * n_seg));
    return locus_launch_status();
}

// n_rows: the rows of `out`, which bound the tokens of all segments together.  At most two a segment (decoding), or no
// more than a lone request of few tokens: the tokens kernel.  Where portions may stand beside single tokens each block of the walk
// looks at its own request: a prompt portion of 100 tokens beside 32 decoding requests, 16 heads of 128, takes 41 us;
// all of it in tiles took 107, all of it token by token 55.
extern "C" int locus_delta_scan(const float* q, int ldq, int off_q, const float* k, int ldk, int off_k, const float* v, int ldv,
                                int off_v, const float* beta, const float* decay, float* state, long long slot_stride,
                                const int* state_slots, const int* seg_q0, const int* seg_qn, int n_seg, int n_rows, float* out,
                                int ldo, int H, int heads_per_group, int d, int dv, cudaStream_t stream) {
    if (n_seg <= 0) return 0;
    if (H <= 0 || heads_per_group <= 0 || H % heads_per_group || d <= 0 || d > 256 || dv <= 0 || n_seg > 65535)
        return LOCUS_ERR_UNSUPPORTED;
    DeltaArgs a;
    a.q = q; a.k = k; a.v = v; a.beta = beta; a.decay = decay; a.state = state; a.state_slots = state_slots;
    a.seg_q0 = seg_q0; a.seg_qn = seg_qn; a.out = out; a.slot_stride = slot_stride; a.ldq = ldq; a.off_q = off_q;
    a.ldk = ldk; a.off_k = off_k; a.ldv = ldv; a.off_v = off_v; a.ldo = ldo; a.H = H; a.heads_per_group = heads_per_group;
    a.d = d; a.dv = dv;
    if (walk_not_needed(n_rows, n_seg, d)) {
        const int col_blocks = (dv + 15) / 16;
        const dim3 grid(H * col_blocks, n_seg);
        if (d <= 32) locus_launch(delta_tokens_kernel<4>, grid, dim3(128), 0, stream, a, col_blocks);
        else if (d <= 64) locus_launch(delta_tokens_kernel<8>, grid, dim3(128), 0, stream, a, col_blocks);
        else if (d <= 128) locus_launch(delta_tokens_kernel<16>, grid, dim3(128), 0, stream, a, col_blocks);
        else locus_launch(delta_tokens_kernel<32>, grid, dim3(128), 0, stream, a, col_blocks);
        return locus_launch_status();
    }
    const bool mixed = walk_may_be_mixed(n_rows, n_seg);
    const bool vec = ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k)) & 15) == 0 &&
                     ((ldq | off_q | ldk | off_k | d) & 3) == 0;
    if (d <= 64) return mixed ? delta_walk<2, true>(a, vec, n_seg, stream) : delta_walk<2, false>(a, vec, n_seg, stream);
    if (d <= 128) return mixed ? delta_walk<4, true>(a, vec, n_seg, stream) : delta_walk<4, false>(a, vec, n_seg, stream);
    return mixed ? delta_walk<8, true>(a, vec, n_seg, stream) : delta_walk<8, false>(a, vec, n_seg, stream);
}

__device__ __forceinline__ float dr_silu(float x) { return x / (1.0f + expf(-x)); }

// One warp per (token, head).
template <typename TO>
__global__ void __launch_bounds__(256) delta_out_kernel(const float* __restrict__ o, const float* __restrict__ proj, int ld,
                                                        int off_g, const void* __restrict__ w, int w_dt, int w_len, float eps,
                                                        TO* __restrict__ out, int n_units, int H, int dv) {
    pdl_entry();
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const int unit = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (unit >= n_units) return;
    const int t = unit / H, h = unit % H;
    const float* orow = o + (static_cast<size_t>(t) * H + h) * dv;
    const float* grow = proj + static_cast<size_t>(t) * ld + off_g + h * dv;
    float ss = 0.f;
    for (int j = lane; j < dv; j += 32) ss = fmaf(orow[j], orow[j], ss);
    ss = warp_sum(ss);
    const float scale = 1.0f / sqrtf(ss / static_cast<float>(dv) + eps);
    TO* dst = out + (static_cast<size_t>(t) * H + h) * dv;
    for (int j = lane; j < dv; j += 32)
        dst[j] = from_f<TO>(orow[j] * scale * ld_dyn(w, w_dt, (h * dv + j) % w_len) * dr_silu(grow[j]));
}

// o [T, H * dv] float32; the gate's columns [off_g, off_g + H * dv) of proj [T, ld] float32; w [w_len] with w_len = dv
// (one weight for all heads) or H * dv; out [T, H * dv].
extern "C" int locus_delta_out(const float* o, const float* proj, int ld, int off_g, const void* w, int w_dt, int w_len,
                               float eps, void* out, int out_dt, int T, int H, int dv, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (H <= 0 || dv <= 0 || (w_len != dv && w_len != H * dv)) return LOCUS_ERR_UNSUPPORTED;
    const long long units = static_cast<long long>(T) * H;
    if (units > 0x7fffffffLL) return LOCUS_ERR_UNSUPPORTED;
    const int n = static_cast<int>(units), blocks = (n + 7) / 8;
    if (out_dt == LOCUS_DT_BF16)
        locus_launch(delta_out_kernel<bf16>, dim3(blocks), dim3(256), 0, stream, o, proj, ld, off_g, w, w_dt, w_len, eps,
                     static_cast<bf16*>(out), n, H, dv);
    else if (out_dt == LOCUS_DT_F32)
        locus_launch(delta_out_kernel<float>, dim3(blocks), dim3(256), 0, stream, o, proj, ld, off_g, w, w_dt, w_len, eps,
                     static_cast<float*>(out), n, H, dv);
    else
        return LOCUS_ERR_UNSUPPORTED;
    return locus_launch_status();
}
