// Matrix products for a handful of rows (decode steps): out[m, n] = sum_k x[m, k] W[n, k],
// at most 8 rows of x per tile.  The work is bound by reading W once from HBM, so the layout
// is that of a matrix-vector product: one warp per output column n streams the weight row
// W[n, :] with 16-byte loads (four in flight per lane), multiplies it with up to 8 rows of x
// (read through L1; they are shared by every warp) in float32, reduces across the warp and
// runs the epilogue.  Same epilogues and the same gathered / grouped forms as the other
// products: bias, SwiGLU of two weight rows, per-row scale, store or add into float32.
//
// The order of an element's sum follows from the kernel and from K (f32_stream: and N) alone (8-element chunks per lane, lanes
// combined by a fixed shuffle tree); what the other rows hold never matters.  Which kernel runs follows from the number of rows:
// float32 rows of one or two (grouped: up to 8 pairs), of 3 to 32 and of more round differently from one another.
//
// float32 x float32 has a kernel of its own, f32_stream: with a warp per weight row every 16 bytes of a weight row cost the 8
// rows' 128 bytes of x from L1, which was the bound (2.5 TB/s of weights).  There a warp streams four weight rows, so that a
// piece of x serves all four; a lane's products are summed over even and odd k, and the lanes' sums change hands as in
// walk.cuh.  The weights arrive by asynchronous copies, two pieces of 128 floats of each row ahead (held in registers a
// second piece spilled: 3.8 TB/s on the head).  Where a plain product has few weight rows (fewer than 20,000: 5,000 warps, two
// rounds of the 16 that an SM holds) two, four or eight warps share K in pieces and their shares are added in order, the
// number following from N and K alone.  Measured at 8 rows: 151,936 x 2,048 264 us = 4.7 TB/s, 6,144 x 2,048 19.4 us (39.7
// before), the routed experts of 8 tokens 141 us = 5.9 TB/s (192 before).  More rows run in tiles of 8 that find the weights in
// L2, where that is quicker than gemm_simt.cu (kernels/__init__.py: F32_STREAM_ANY).  One or two rows stay on the warp-per-row kernel (11.0 us
// against 13.4 at one row), and so do grouped products of up to 8 rows, whose few tiles hold a row each (a decode step of
// one request, 24 layers of 60 experts with 4 picks: 3.20 ms against 3.49).
#include "common.cuh"
#include "walk.cuh"

#define GV_ROWS 8    // rows of x per tile
#define GV_WARPS 8   // output columns per block

struct GemvArgs {
    const void* x;
    const void* w;
    const void* w2;
    const void* bias;
    int bias_dt;
    void* out;
    int out_dt;
    int accumulate;
    int act;  // 1: relu(v)^2 after the bias, before the row scale; 2 (two weights): the clamped gated unit of gemm_simt.cu;
              // 3 (one weight): act_param tanh(act_scale v / act_param), behind everything else
              // 4 (two weights): relu(v + b) (u + b2), then the row scale (`bias` is [2N]: b and behind it b2)
    float act_param, act_scale;
    const float* row_scale;
    const int* scale_rows;
    const int* x_rows;
    int x_row_div;
    int M, N, K;
    long long ldx, ldo;
    const int* tile_expert;
    const int* tile_row0;
    const int* tile_rows;
    const int* n_tiles;
    long long w_expert_stride;
};

template <typename T>
__device__ __forceinline__ void load8(const T* p, float* o);
template <>
__device__ __forceinline__ void load8<float>(const float* p, float* o) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
}
template <>
__device__ __forceinline__ void load8<bf16>(const bf16* p, float* o) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(h[i]);
        o[2 * i] = f.x;
        o[2 * i + 1] = f.y;
    }
}

// streaming load of weights: read once, do not keep in L1
template <typename T>
__device__ __forceinline__ void load8_stream(const T* p, float* o);
template <>
__device__ __forceinline__ void load8_stream<float>(const float* p, float* o) {
    const float4 a = __ldcs(reinterpret_cast<const float4*>(p)), b = __ldcs(reinterpret_cast<const float4*>(p + 4));
    o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
}
template <>
__device__ __forceinline__ void load8_stream<bf16>(const bf16* p, float* o) {
    const uint4 v = __ldcs(reinterpret_cast<const uint4*>(p));
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(h[i]);
        o[2 * i] = f.x;
        o[2 * i + 1] = f.y;
    }
}

template <typename TX, typename TW, bool DUAL, int ROWS>
__device__ __forceinline__ void gemv_body(const GemvArgs& a, const TW* __restrict__ w, const TW* __restrict__ w2,
                                          const TX* const* xr, int rows, int lane, float* acc, float* acc2) {
    const int K = a.K;
    // 8-element chunks, four weight loads in flight per lane
    int j = lane * 8;
    for (; j + 3 * 256 < K; j += 4 * 256) {
        float wv[4][8], uv[DUAL ? 4 : 1][8];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            load8_stream<TW>(w + j + u * 256, wv[u]);
            if (DUAL) load8_stream<TW>(w2 + j + u * 256, uv[u]);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
#pragma unroll
            for (int t = 0; t < ROWS; ++t) {
                if (t < rows) {
                    float hv[8];
                    load8<TX>(xr[t] + j + u * 256, hv);
#pragma unroll
                    for (int v = 0; v < 8; ++v) {
                        acc[t] = fmaf(hv[v], wv[u][v], acc[t]);
                        if (DUAL) acc2[t] = fmaf(hv[v], uv[u][v], acc2[t]);
                    }
                }
            }
        }
    }
    for (; j < K; j += 256) {
        float wv[8], uv[8];
        load8_stream<TW>(w + j, wv);
        if (DUAL) load8_stream<TW>(w2 + j, uv);
#pragma unroll
        for (int t = 0; t < ROWS; ++t) {
            if (t < rows) {
                float hv[8];
                load8<TX>(xr[t] + j, hv);
#pragma unroll
                for (int v = 0; v < 8; ++v) {
                    acc[t] = fmaf(hv[v], wv[v], acc[t]);
                    if (DUAL) acc2[t] = fmaf(hv[v], uv[v], acc2[t]);
                }
            }
        }
    }
}

// One output: activation, bias, row scale (rs), softcap, store.  u: the second weight's sum.
template <bool DUAL>
__device__ __forceinline__ void gemv_store(const GemvArgs& a, int r, int n, float rs, float v, float u) {
    if (DUAL && a.act == 2) {
        const float g = fminf(v * rs, a.act_param), uc = fminf(fmaxf(u * rs, -a.act_param), a.act_param);
        v = g / (1.0f + expf(-1.702f * g)) * (uc + 1.0f);
    } else if (DUAL && a.act == 4) {
        v = fmaxf(v + pair_bias(a.bias, a.bias_dt, n), 0.f) * (u + pair_bias(a.bias, a.bias_dt, a.N + n));
    } else if (DUAL) {
        v = v / (1.0f + expf(-v)) * u;
    }
    if (a.bias && a.act != 4) v += ld_dyn(a.bias, a.bias_dt, n);
    if (a.act == 1) {
        v = fmaxf(v, 0.f);
        v *= v;
    }
    if (a.row_scale && a.act != 2) v *= rs;
    if (a.act == 3) v = a.act_param * tanhf(v * a.act_scale / a.act_param);
    const size_t o = static_cast<size_t>(r) * a.ldo + n;
    if (a.accumulate) {
        static_cast<float*>(a.out)[o] += v;
    } else {
        st_dyn(a.out, a.out_dt, o, v);
    }
}

template <typename TX, typename TW, bool DUAL>
__global__ void __launch_bounds__(32 * GV_WARPS) rowstream_kernel(GemvArgs a) {
    int row0, rows;
    const TW* W = static_cast<const TW*>(a.w);
    const TW* W2 = static_cast<const TW*>(a.w2);
    if (a.tile_expert != nullptr) {
        const int tile = blockIdx.y;
        if (tile >= *a.n_tiles) return;
        const long long e = a.tile_expert[tile];
        row0 = a.tile_row0[tile];
        rows = a.tile_rows[tile];
        W += e * a.w_expert_stride;
        if (DUAL) W2 += e * a.w_expert_stride;
    } else {
        row0 = blockIdx.y * GV_ROWS;
        rows = min(GV_ROWS, a.M - row0);
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int n = blockIdx.x * GV_WARPS + wid;
    if (n >= a.N) return;
    const TX* xr[GV_ROWS];
#pragma unroll
    for (int t = 0; t < GV_ROWS; ++t) {
        const int r = row0 + (t < rows ? t : 0);
        const long long xrow = a.x_rows ? a.x_rows[r] / a.x_row_div : r;
        xr[t] = static_cast<const TX*>(a.x) + xrow * a.ldx;
    }
    float acc[GV_ROWS], acc2[GV_ROWS];
#pragma unroll
    for (int t = 0; t < GV_ROWS; ++t) acc[t] = acc2[t] = 0.f;
    const TW* w = W + static_cast<long long>(n) * a.K;
    const TW* w2 = DUAL ? W2 + static_cast<long long>(n) * a.K : nullptr;
    // fewer unrolled rows when the tile is small keeps registers and instructions down
    if (rows == 1) gemv_body<TX, TW, DUAL, 1>(a, w, w2, xr, rows, lane, acc, acc2);
    else if (rows <= 2) gemv_body<TX, TW, DUAL, 2>(a, w, w2, xr, rows, lane, acc, acc2);
    else if (rows <= 4) gemv_body<TX, TW, DUAL, 4>(a, w, w2, xr, rows, lane, acc, acc2);
    else gemv_body<TX, TW, DUAL, GV_ROWS>(a, w, w2, xr, rows, lane, acc, acc2);
#pragma unroll
    for (int t = 0; t < GV_ROWS; ++t) {
        if (t >= rows) break;
        float v = warp_sum(acc[t]);
        float u = DUAL ? warp_sum(acc2[t]) : 0.f;
        if (lane != 0) continue;
        const int r = row0 + t;
        const float rs = a.row_scale ? a.row_scale[a.scale_rows ? a.scale_rows[r] : r] : 1.0f;
        gemv_store<DUAL>(a, r, n, rs, v, u);
    }
}

#define GV_NC 4       // weight rows of a warp of f32_stream (with DUAL two of each weight)
#define GV_STAGES 3   // pieces of 128 floats of them that are on their way or worked on

// ROWS: rows of x that are worked on (a tile's rows are at most that).  `share` of `split`: this warp's pieces of K.
// ring: this lane's 16 bytes of every weight row and stage, 512 bytes apart: a lane reads only what it copied itself.
// shares: [GV_WARPS][GV_NC * GV_ROWS] floats of shared memory.
template <int ROWS, bool DUAL>
__device__ __forceinline__ void f32_stream_body(const GemvArgs& a, const float* W, const float* W2, int row0, int rows, int n0,
                                                int share, int split, bool wait, float* ring, float (*shares)[GV_NC * GV_ROWS]) {
    constexpr int NC = GV_NC, COLS = DUAL ? NC / 2 : NC, V = ROWS * NC;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const float* w[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const int n = min(n0 + c % COLS, a.N - 1);   // (a weight row behind the last: the last one again, its sum unused)
        w[c] = (DUAL && c >= COLS ? W2 : W) + static_cast<long long>(n) * a.K;
    }
    const int k0 = 128 * share + 4 * lane, step = 128 * split;
    const int n_pieces = (a.K - 128 * share + step - 1) / step;   // (the same for all lanes of a warp; may be 0 or less)
    auto fetch = [&](int i) {
        if (i < n_pieces) {
            const int k = k0 + i * step;
            const bool live = k < a.K;
#pragma unroll
            for (int c = 0; c < NC; ++c) walk_copy<16>(ring + ((i % GV_STAGES) * NC + c) * 128, w[c] + (live ? k : 0), live);
        }
        walk_commit();
    };
#pragma unroll
    for (int i = 0; i < GV_STAGES - 1; ++i) fetch(i);
    if (wait) pdl_entry();   // the first weights are on their way before the kernel in front has finished
    const float* x[ROWS];
#pragma unroll
    for (int t = 0; t < ROWS; ++t) {
        const int r = row0 + (t < rows ? t : 0);
        x[t] = static_cast<const float*>(a.x) + (a.x_rows ? a.x_rows[r] / a.x_row_div : r) * a.ldx;
    }
    f2 acc[NC][ROWS];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int t = 0; t < ROWS; ++t) acc[c][t] = 0;
    for (int i = 0; i < n_pieces; ++i) {
        const int k = k0 + i * step;
        fetch(i + GV_STAGES - 1);
        walk_wait<GV_STAGES - 1>();
        ulonglong2 wv[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) wv[c] = *reinterpret_cast<const ulonglong2*>(ring + ((i % GV_STAGES) * NC + c) * 128);
        if (k < a.K) {
#pragma unroll
            for (int t = 0; t < ROWS; ++t) {
                const ulonglong2 xv = *reinterpret_cast<const ulonglong2*>(x[t] + k);   // (a row that is not there: the first one)
#pragma unroll
                for (int c = 0; c < NC; ++c) acc[c][t] = f2_fma(wv[c].y, xv.y, f2_fma(wv[c].x, xv.x, acc[c][t]));
            }
        }
    }
    pdl_trigger();
    float sums[V];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int t = 0; t < ROWS; ++t) {
            float e, f;
            f2_unpack(acc[c][t], e, f);
            sums[c * ROWS + t] = e + f;
        }
    const float sum = walk_sum<V>(sums, lane);
    if (lane < V) shares[wid][walk_sum_index<V>(lane)] = sum;
    __syncthreads();
    const int c = lane / ROWS, t = lane % ROWS, n = n0 + c;
    if (share != 0 || lane >= COLS * ROWS || t >= rows || n >= a.N) return;
    float v = 0.f, u = 0.f;
    for (int j = 0; j < split; ++j) {
        v += shares[wid + j][lane];
        if (DUAL) u += shares[wid + j][COLS * ROWS + lane];
    }
    const int r = row0 + t;
    const float rs = a.row_scale ? a.row_scale[a.scale_rows ? a.scale_rows[r] : r] : 1.0f;
    gemv_store<DUAL>(a, r, n, rs, v, u);
}

// Grid (tiles of 8 rows, blocks of weight rows, and again): the tiles of the same weights run together, so that a second tile finds them
// in L2; the blocks go on along the third index, since 65,535 along the second hold 2.1 million rows.
template <bool DUAL>
__global__ void __launch_bounds__(32 * GV_WARPS, 2) f32_stream_kernel(GemvArgs a, int split) {
    extern __shared__ __align__(16) float ring_smem[];   // [warp][stage][weight row][128]
    __shared__ float shares[GV_WARPS][GV_NC * GV_ROWS];
    const float* W = static_cast<const float*>(a.w);
    const float* W2 = static_cast<const float*>(a.w2);
    int row0, rows;
    const bool grouped = a.tile_expert != nullptr;
    const int tile = blockIdx.x, block = blockIdx.z * gridDim.y + blockIdx.y;
    if (grouped) {
        pdl_entry();   // (the lists come from the kernels in front)
        if (tile >= *a.n_tiles) return;
        const long long e = a.tile_expert[tile];
        row0 = a.tile_row0[tile];
        rows = a.tile_rows[tile];
        W += e * a.w_expert_stride;
        if (DUAL) W2 += e * a.w_expert_stride;
    } else {
        row0 = tile * GV_ROWS;
        rows = min(GV_ROWS, a.M - row0);
    }
    const int wid = threadIdx.x >> 5;
    const int n0 = (block * (GV_WARPS / split) + wid / split) * (DUAL ? GV_NC / 2 : GV_NC);
    float* ring = ring_smem + wid * GV_STAGES * GV_NC * 128 + (threadIdx.x & 31) * 4;
    if (rows <= 2) f32_stream_body<2, DUAL>(a, W, W2, row0, rows, n0, wid % split, split, !grouped, ring, shares);
    else if (rows <= 4) f32_stream_body<4, DUAL>(a, W, W2, row0, rows, n0, wid % split, split, !grouped, ring, shares);
    else f32_stream_body<8, DUAL>(a, W, W2, row0, rows, n0, wid % split, split, !grouped, ring, shares);
}

static int launch_f32(const GemvArgs& a, int tiles, bool dual, cudaStream_t stream) {
    const int groups = ceil_div(a.N, dual ? GV_NC / 2 : GV_NC);   // four weight rows each
    int split = 1;
    while (a.tile_expert == nullptr && split < GV_WARPS && groups * split < 5000 && a.K >= 256 * split) split *= 2;
    const int blocks = ceil_div(groups, GV_WARPS / split), layers = ceil_div(blocks, 65535);
    const dim3 grid(tiles, layers > 0 ? ceil_div(blocks, layers) : 0, layers);
    if (grid.x == 0 || grid.y == 0) return 0;
    constexpr size_t smem = sizeof(float) * GV_WARPS * GV_STAGES * GV_NC * 128;
    auto* kernel = dual ? f32_stream_kernel<true> : f32_stream_kernel<false>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    locus_launch(kernel, grid, dim3(32 * GV_WARPS), smem, stream, a, split);
    return locus_launch_status();
}

template <typename TX, typename TW>
static int launch(const GemvArgs& a, int tiles, bool dual, cudaStream_t stream) {
    dim3 grid(ceil_div(a.N, GV_WARPS), tiles);
    if (grid.x == 0 || grid.y == 0) return 0;
    if (grid.y > 65535) return LOCUS_ERR_UNSUPPORTED;
    if (dual) {
        rowstream_kernel<TX, TW, true><<<grid, 32 * GV_WARPS, 0, stream>>>(a);
    } else {
        rowstream_kernel<TX, TW, false><<<grid, 32 * GV_WARPS, 0, stream>>>(a);
    }
    return locus_launch_status();
}

// Same arguments as locus_gemm_simt.  Needs K a multiple of 8, rows of x and W that start on
// 16-byte (bfloat16) / 32-byte (float32) boundaries, and, for a grouped product, tiles of at
// most 8 rows.
extern "C" int locus_gemv(const void* x, int x_dt, const void* w, const void* w2, int w_dt, const void* bias,
                          int bias_dt, void* out, int out_dt, int flags, float act_param, float act_scale, const float* row_scale,
                          const int* scale_rows, const int* x_rows, int x_row_div, int M, int N, int K,
                          long long ldx, long long ldo, const int* tile_expert, const int* tile_row0,
                          const int* tile_rows, const int* n_tiles, int max_tiles, long long w_expert_stride,
                          cudaStream_t stream) {
    if (N <= 0 || K <= 0 || K % 8 != 0 || ldx % 8 != 0) return LOCUS_ERR_UNSUPPORTED;
    const int accumulate = flags & 1, act = (flags >> 1) & 7;  // the flags of locus_gemm_simt
    if ((act == 1 && w2 != nullptr) || ((act == 2 || act == 4) && w2 == nullptr) || act > 4 || (act == 3 && (w2 != nullptr || !(act_param > 0.f)))) return LOCUS_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(w2)) & 31)
        return LOCUS_ERR_UNSUPPORTED;
    if (accumulate && out_dt != LOCUS_DT_F32) return LOCUS_ERR_UNSUPPORTED;
    if (x_rows != nullptr && x_row_div <= 0) return LOCUS_ERR_UNSUPPORTED;
    GemvArgs a;
    a.x = x; a.w = w; a.w2 = w2; a.bias = bias; a.bias_dt = bias_dt; a.out = out; a.out_dt = out_dt;
    a.accumulate = accumulate; a.act = act; a.act_param = act_param; a.act_scale = act_scale; a.row_scale = row_scale; a.scale_rows = scale_rows; a.x_rows = x_rows;
    a.x_row_div = x_row_div; a.M = M; a.N = N; a.K = K; a.ldx = ldx; a.ldo = ldo;
    a.tile_expert = tile_expert; a.tile_row0 = tile_row0; a.tile_rows = tile_rows; a.n_tiles = n_tiles;
    a.w_expert_stride = w_expert_stride;
    const int tiles = tile_expert ? max_tiles : ceil_div(M, GV_ROWS);
    const bool dual = w2 != nullptr;
    if (x_dt == LOCUS_DT_F32 && w_dt == LOCUS_DT_F32)
        return M <= (tile_expert == nullptr ? 2 : 8) ? launch<float, float>(a, tiles, dual, stream) : launch_f32(a, tiles, dual, stream);
    if (x_dt == LOCUS_DT_BF16 && w_dt == LOCUS_DT_BF16) return launch<bf16, bf16>(a, tiles, dual, stream);
    if (x_dt == LOCUS_DT_BF16 && w_dt == LOCUS_DT_F32) return launch<bf16, float>(a, tiles, dual, stream);
    if (x_dt == LOCUS_DT_F32 && w_dt == LOCUS_DT_BF16) return launch<float, bf16>(a, tiles, dual, stream);
    return LOCUS_ERR_UNSUPPORTED;
}
