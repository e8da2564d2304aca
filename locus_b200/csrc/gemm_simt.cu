// Matrix products on CUDA cores with float32 FMA: out = x . W^T with fused epilogues.
//
// This is the true-32-bit path of the linear layers whose work is too small for gemm_f32_tc.cuh (float32 on the tensor cores, no
// TF32: the choice is f32_tc_takes in kernels/__init__.py) and the general fallback of the bfloat16 path for shapes the
// tensor-core kernels refuse.  In
// gemm_simt one thread accumulates an output over k = 0..K-1 in ascending order, so its value
// does not depend on M, on the other rows of the batch or on the tile it falls in.  In gemm_f32
// an output is a sum over the even k and one over the odd k, and a plain product may be cut
// along K, by M, N and K: the other rows' values never matter, but a row of M rows may round
// otherwise than the same row among more or fewer, whose product is cut otherwise or runs on
// gemv.cu.
//
// Both kernels cover:
//   * plain      out[m, n]  = sum_k x[m, k] W[n, k]          (+ bias[n]) (* row_scale[m])
//   * SwiGLU     out[m, n]  = silu(x . Wg[n]) * (x . Wu[n])   (two accumulators)
//   * gathered   x row of logical row m is x_rows[m] / x_row_div
//   * grouped    logical rows are sorted by expert; a device-built tile list names, for
//                each 64-row tile, its expert, first row and row count; W of expert e
//                starts at W + e * w_expert_stride
//   * epilogue   store as float32 or bfloat16, or add into a float32 tensor (residual)
//
// Two kernels.  gemm_f32: float32 rows and weights that 16-byte copies can fetch.  Bound by the multiply-adds (148 SMs x 128
// lanes x 2 x 1.965 GHz = 74.4 TFLOP/s), so everything else is kept off their issue slots: 32 columns of k of 64 rows
// and 128 weight rows are copied into shared memory asynchronously, two stages ahead, k contiguous as they lie in memory (rows
// 36 floats apart meet in no bank), a thread owns 8 x 8 outputs, and a multiply-add works on two k at once, so each
// output has a sum over the even k and one over the odd k, added at the end; a product whose blocks would leave SMs idle is
// cut along k, its parts added up in order by a second kernel.  A tile's rows are worked on in eights, so that an expert's 34
// rows cost 40 and not 64.  gemm_simt: every other type, width and alignment.  Measured: 2,048 x 6,144 x 2,048 1.16 ms = 44.6
// TFLOP/s (2.0 ms with the 64 x 64 x 16 tiles of gemm_simt), 512 x 6,144 x 2,048 302 us, 64 x 512 x 512 10 us, the routed experts
// of 512 tokens (60 x (2,048 -> 1,408 -> 2,048), 4 picks) 1.01 ms; one multiply-add at a time instead of two, with up to twice the
// warps, 1.26 to 1.5 ms on the first.
#include "common.cuh"
#include "walk.cuh"

#define BM 64
#define BN 64
#define BK 16

struct GemmArgs {
    const void* x;
    const void* w;
    const void* w2;          // up-projection for SwiGLU, else null
    const void* bias;        // [N] or null
    int bias_dt;
    void* out;
    int out_dt;
    int accumulate;          // out (float32) += result
    int act;                 // 0: none; 1: relu(v)^2 (after the bias, before the row scale); 2 (with w2): the clamped
                             // gated unit g' sigmoid(1.702 g') (u' + 1), g' = min(s g, limit), u' = clamp(s u, +-limit),
                             // s the row's scale, which then stands for a factor on the input; 4 (with w2): relu(v + b) (u + b2),
                             // then the row scale (`bias` is [2N]: b and behind it b2)
    float act_param;         // the limit of act 2; the cap of act 3 (without w2): cap tanh(act_scale v / cap), behind everything else
    float act_scale;
    const float* row_scale;  // or null: row m is scaled by row_scale[scale_rows ? scale_rows[m] : m]
    const int* scale_rows;
    const int* x_rows;       // [M] or null
    int x_row_div;
    int M, N, K;
    long long ldx, ldo;
    // grouped
    const int* tile_expert;  // null when not grouped
    const int* tile_row0;
    const int* tile_rows;
    const int* n_tiles;
    long long w_expert_stride;
    // gemm_f32, plain products cut along K: [splits][M][N] sums that gemm_f32_sum adds up in order (null: not cut)
    float* part;
    int splits;
};

// One output: activation, bias (b; of the second weight b2), row scale (rs), softcap.  v2: the second weight's sum.
template <bool SWIGLU>
__device__ __forceinline__ float finish(const GemmArgs& a, float rs, float v, float v2, float b, float b2) {
    if (SWIGLU && a.act == 2) {
        const float g = fminf(v * rs, a.act_param);
        const float u = fminf(fmaxf(v2 * rs, -a.act_param), a.act_param);
        v = g / (1.0f + expf(-1.702f * g)) * (u + 1.0f);
    } else if (SWIGLU && a.act == 4) {
        v = fmaxf(v + b, 0.f) * (v2 + b2);
    } else if (SWIGLU) {
        const float g = v;
        v = g / (1.0f + expf(-g)) * v2;
    }
    if (a.bias && a.act != 4) v += b;
    if (a.act == 1) {
        v = fmaxf(v, 0.f);
        v *= v;
    }
    if (a.row_scale && a.act != 2) v *= rs;
    if (a.act == 3) v = a.act_param * tanhf(v * a.act_scale / a.act_param);
    return v;
}
__device__ __forceinline__ float bias_of(const GemmArgs& a, int n) { return pair_bias(a.bias, a.bias_dt, n); }
__device__ __forceinline__ float scale_of(const GemmArgs& a, int r) {
    return a.row_scale ? a.row_scale[a.scale_rows ? a.scale_rows[r] : r] : 1.0f;
}

// The same, stored or added, for the kernels that unroll it over a thread's outputs (with the biases in hand it ran 2 us longer).
template <bool SWIGLU>
__device__ __forceinline__ void epilogue(const GemmArgs& a, int r, int n, float rs, float v, float v2) {
    if (SWIGLU && a.act == 2) {
        const float g = fminf(v * rs, a.act_param);
        const float u = fminf(fmaxf(v2 * rs, -a.act_param), a.act_param);
        v = g / (1.0f + expf(-1.702f * g)) * (u + 1.0f);
    } else if (SWIGLU && a.act == 4) {
        v = fmaxf(v + pair_bias(a.bias, a.bias_dt, n), 0.f) * (v2 + pair_bias(a.bias, a.bias_dt, a.N + n));
    } else if (SWIGLU) {
        const float g = v;
        v = g / (1.0f + expf(-g)) * v2;
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

template <typename TX, typename TW, bool SWIGLU>
__global__ void __launch_bounds__(256) gemm_simt_kernel(GemmArgs a) {
    __shared__ float xs[BK][BM + 4];
    __shared__ float ws[BK][BN + 4];
    __shared__ float ws2[SWIGLU ? BK : 1][BN + 4];

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
        if (SWIGLU) W2 += e * a.w_expert_stride;
    } else {
        row0 = blockIdx.y * BM;
        rows = min(BM, a.M - row0);
    }
    const int col0 = blockIdx.x * BN;
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;  // 16 x 16 threads, 4 x 4 outputs each
    const TX* X = static_cast<const TX*>(a.x);

    // loader mapping: thread loads elements (lr, lk..lk+3) of the x tile and of the W tile
    const int lr = tid >> 2, lk = (tid & 3) * 4;
    long long xrow = -1;
    if (lr < rows) {
        const int r = row0 + lr;
        xrow = a.x_rows ? a.x_rows[r] / a.x_row_div : r;
    }
    const int wrow = col0 + lr;

    float acc[4][4], acc2[SWIGLU ? 4 : 1][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            acc[i][j] = 0.f;
            if (SWIGLU) acc2[i][j] = 0.f;
        }

    for (int k0 = 0; k0 < a.K; k0 += BK) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = k0 + lk + u;
            float xv = 0.f, wv = 0.f, wv2 = 0.f;
            if (k < a.K) {
                if (xrow >= 0) xv = to_f(X[xrow * a.ldx + k]);
                if (wrow < a.N) {
                    wv = to_f(W[static_cast<long long>(wrow) * a.K + k]);
                    if (SWIGLU) wv2 = to_f(W2[static_cast<long long>(wrow) * a.K + k]);
                }
            }
            xs[lk + u][lr] = xv;
            ws[lk + u][lr] = wv;
            if (SWIGLU) ws2[lk + u][lr] = wv2;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float av[4], bv[4], bv2[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) av[i] = xs[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                bv[j] = ws[kk][tx * 4 + j];
                if (SWIGLU) bv2[j] = ws2[kk][tx * 4 + j];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
                    if (SWIGLU) acc2[i][j] = fmaf(av[i], bv2[j], acc2[i][j]);
                }
        }
        __syncthreads();
    }

#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int lrow = ty * 4 + i;
        if (lrow >= rows) continue;
        const int r = row0 + lrow;
        const float rs = a.row_scale ? a.row_scale[a.scale_rows ? a.scale_rows[r] : r] : 1.0f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = col0 + tx * 4 + j;
            if (n < a.N) epilogue<SWIGLU>(a, r, n, rs, acc[i][j], SWIGLU ? acc2[i][j] : 0.f);
        }
    }
}

#define FM 64          // rows of a tile
#define FK 32          // columns of k of a stage
#define FLD (FK + 4)   // floats from row to row of a stage
#define F_STAGES 3

// A stage's share of eight-row groups 0 .. NI - 1: thread (ty, tx) owns the rows ty + 8 i and the weight rows tx + TX j.
template <int NI, int TX>
__device__ __forceinline__ void f32_stage(const float* xs, const float* ws, f2 (&acc)[8][8]) {
#pragma unroll
    for (int k = 0; k < FK; k += 4) {
        ulonglong2 x[NI];
#pragma unroll
        for (int i = 0; i < NI; ++i) x[i] = *reinterpret_cast<const ulonglong2*>(xs + 8 * i * FLD + k);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(ws + TX * j * FLD + k);
#pragma unroll
            for (int i = 0; i < NI; ++i) acc[i][j] = f2_fma(x[i].x, w.x, acc[i][j]);
#pragma unroll
            for (int i = 0; i < NI; ++i) acc[i][j] = f2_fma(x[i].y, w.y, acc[i][j]);
        }
    }
}

// TX: threads across the weight rows of a tile (8 TX of them; with SWIGLU 4 TX of each weight).
template <int TX, bool SWIGLU>
__global__ void __launch_bounds__(8 * TX) gemm_f32_kernel(GemmArgs a) {
    constexpr int BNW = 8 * TX, COLS = SWIGLU ? BNW / 2 : BNW, NT = 8 * TX, STAGE = (FM + BNW) * FLD;
    extern __shared__ __align__(16) float f32_smem[];
    int row0, rows;
    const float* W = static_cast<const float*>(a.w);
    const float* W2 = static_cast<const float*>(a.w2);
    if (a.tile_expert != nullptr) {
        const int tile = blockIdx.y;
        if (tile >= *a.n_tiles) return;
        const long long e = a.tile_expert[tile];
        row0 = a.tile_row0[tile];
        rows = a.tile_rows[tile];
        W += e * a.w_expert_stride;
        if (SWIGLU) W2 += e * a.w_expert_stride;
    } else {
        row0 = blockIdx.y * FM;
        rows = min(FM, a.M - row0);
    }
    const int col0 = blockIdx.x * COLS, tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    // the copies of this thread: 16 bytes of k (chunk tid & 7) of every NT / 8-th row
    constexpr int PER = NT / 8;
    const int chunk = (tid & 7) * 4, lrow = tid >> 3;
    int xrow[FM / PER];
#pragma unroll
    for (int i = 0; i < FM / PER; ++i) {
        const int r = row0 + lrow + i * PER;
        xrow[i] = lrow + i * PER >= rows ? -1 : a.x_rows ? a.x_rows[r] / a.x_row_div : r;
    }
    const int n_all = (a.K + FK - 1) / FK, per_split = (n_all + a.splits - 1) / a.splits;
    const int kb0 = blockIdx.z * per_split, n_k = min(per_split, n_all - kb0), live_rows = (rows + 7) & ~7;
    auto fetch = [&](int kb) {   // columns behind K and rows that are not there are zeros
        float* st = f32_smem + (kb % F_STAGES) * STAGE + lrow * FLD + chunk;
        const int k = (kb0 + kb) * FK + chunk;
        const bool in = k < a.K;
#pragma unroll
        for (int i = 0; i < FM / PER; ++i)
            if (lrow + i * PER < live_rows) {
                const bool live = in && xrow[i] >= 0;
                walk_copy<16>(st + i * PER * FLD, live ? static_cast<const float*>(a.x) + xrow[i] * a.ldx + k : W, live);
            }
#pragma unroll
        for (int i = 0; i < BNW / PER; ++i) {
            const int c = lrow + i * PER, n = col0 + (SWIGLU ? c % COLS : c);
            const bool live = in && n < a.N;
            const float* w = SWIGLU && i * PER >= COLS ? W2 : W;   // (COLS is a multiple of PER)
            walk_copy<16>(st + (FM + i * PER) * FLD, live ? w + static_cast<long long>(n) * a.K + k : W, live);
        }
    };
    f2 acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0;
#pragma unroll
    for (int i = 0; i < F_STAGES - 1; ++i) {
        if (i < n_k) fetch(i);
        walk_commit();
    }
    // An instance each for 2, 4, 5, 6 and 8 eights of rows, the next larger one for the others.  With three more, for 1, 3 and 7, two
    // registers spilled: 24 rows of 6,144 x 2,048 28.1 -> 24.5 us, the experts of 240 tokens 800 -> 748, but those of 512 1,005 ->
    // 1,024 and 2,048 rows 1,155 -> 1,181.
    const int groups = (rows + 7) >> 3;
    auto walk_k = [&](auto stage) {
        for (int kb = 0; kb < n_k; ++kb) {
            walk_wait<F_STAGES - 2>();
            __syncthreads();   // the stage is there for all warps, and nobody reads the one that is filled next
            if (kb + F_STAGES - 1 < n_k) fetch(kb + F_STAGES - 1);
            walk_commit();
            const float* st = f32_smem + (kb % F_STAGES) * STAGE;
            stage(st + ty * FLD, st + (FM + tx) * FLD);
        }
    };
    if (groups <= 2) walk_k([&](const float* x, const float* w) { f32_stage<2, TX>(x, w, acc); });
    else if (groups <= 4) walk_k([&](const float* x, const float* w) { f32_stage<4, TX>(x, w, acc); });
    else if (groups == 5) walk_k([&](const float* x, const float* w) { f32_stage<5, TX>(x, w, acc); });
    else if (groups == 6) walk_k([&](const float* x, const float* w) { f32_stage<6, TX>(x, w, acc); });
    else walk_k([&](const float* x, const float* w) { f32_stage<8, TX>(x, w, acc); });
    // The tile's sums go through shared memory to a loop that holds the epilogue once: unrolled over a thread's 64 outputs its code
    // had to be fetched for a single use, 20 cycles to an instruction (64 x 16 x 64 23 -> 11 us, 512 x 512 x 512 35 -> 21, the
    // routed experts of 300 tokens, 8 x (512 -> 256 -> 512), 89 -> 64).  Old values of an added-to output are fetched together.
    __syncthreads();   // nobody reads the stages any more
    constexpr int LD = BNW + TX;   // (a warp's rows of TX sums meet in no bank)
    float* sums = f32_smem;
    float* olds = sums + FM * LD;
    float* scales = olds + FM * COLS;
    static_assert(FM * (LD + COLS + 1) <= F_STAGES * STAGE, "the epilogue's tile takes the place of the stages");
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float even, odd;
            f2_unpack(acc[i][j], even, odd);
            sums[(ty + 8 * i) * LD + tx + TX * j] = even + odd;
        }
    const int c = tid % COLS, n = col0 + c;
    const bool whole = SWIGLU || a.part == nullptr;
    if (whole && a.accumulate)
        for (int m = tid / COLS; m < rows; m += NT / COLS) {
            const bool live = n < a.N;
            walk_copy<4>(olds + m * COLS + c, static_cast<const float*>(a.out) + static_cast<size_t>(row0 + m) * a.ldo + (live ? n : 0), live);
        }
    walk_commit();
    for (int m = tid; m < rows; m += NT) scales[m] = scale_of(a, row0 + m);
    const float b = n < a.N ? bias_of(a, n) : 0.f, b2 = a.act == 4 && n < a.N ? bias_of(a, a.N + n) : 0.f;
    walk_wait<0>();
    __syncthreads();
    if (n >= a.N) return;
#pragma unroll 2
    for (int m = tid / COLS; m < rows; m += NT / COLS) {
        const float v = sums[m * LD + c];
        if (!whole) {
            a.part[(static_cast<size_t>(blockIdx.z) * a.M + row0 + m) * a.N + n] = v;
            continue;
        }
        const float y = finish<SWIGLU>(a, scales[m], v, SWIGLU ? sums[m * LD + COLS + c] : 0.f, b, b2);
        const size_t o = static_cast<size_t>(row0 + m) * a.ldo + n;
        if (a.accumulate) static_cast<float*>(a.out)[o] = olds[m * COLS + c] + y;
        else st_dyn(a.out, a.out_dt, o, y);
    }
}

// The sums of a product cut along K, in order, and its epilogue.
__global__ void __launch_bounds__(256) gemm_f32_sum_kernel(GemmArgs a) {
    const int n = blockIdx.x * 256 + threadIdx.x, r = blockIdx.y;
    if (n >= a.N) return;
    float v = 0.f;
    for (int z = 0; z < a.splits; ++z) v += a.part[(static_cast<size_t>(z) * a.M + r) * a.N + n];
    epilogue<false>(a, r, n, scale_of(a, r), v, 0.f);
}

#include "gemm_f32_tc.cuh"

template <int TX>
static int launch_f32(const GemmArgs& a, int tiles, bool swiglu, cudaStream_t stream) {
    constexpr size_t smem = sizeof(float) * F_STAGES * (FM + 8 * TX) * FLD;
    const dim3 grid(ceil_div(a.N, swiglu ? 4 * TX : 8 * TX), tiles, a.splits);
    if (grid.y == 0 || grid.x == 0) return 0;
    if (grid.y > 65535) return LOCUS_ERR_UNSUPPORTED;
    auto* kernel = swiglu ? gemm_f32_kernel<TX, true> : gemm_f32_kernel<TX, false>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    kernel<<<grid, 8 * TX, smem, stream>>>(a);
    if (a.part) gemm_f32_sum_kernel<<<dim3(ceil_div(a.N, 256), a.M), 256, 0, stream>>>(a);
    return locus_launch_status();
}

template <typename TX, typename TW>
static int launch(const GemmArgs& a, int max_tiles, bool swiglu, cudaStream_t stream) {
    dim3 grid(ceil_div(a.N, BN), max_tiles);
    if (grid.y == 0 || grid.x == 0) return 0;
    if (grid.y > 65535) return LOCUS_ERR_UNSUPPORTED;
    if (swiglu) {
        gemm_simt_kernel<TX, TW, true><<<grid, 256, 0, stream>>>(a);
    } else {
        gemm_simt_kernel<TX, TW, false><<<grid, 256, 0, stream>>>(a);
    }
    return locus_launch_status();
}

// x_dt / w_dt: element types of x and of W (and W2).  flags: bit 0 = add the result into the float32 out,
// bits 1-3 = the activation: 1 squared ReLU (not with W2), 2 the clamped gated unit with limit act_param (with W2),
// 3 act_param tanh(act_scale v / act_param) (not with W2), 4 relu(x . W + b) (x . W2 + b2) (with W2; bias is then [2N], b and
// behind it b2, or null).  max_tiles: number of 64-row tiles
// to launch; for a grouped product an upper bound (tiles past *n_tiles return at once).  part, splits: a plain product of
// one weight that gemm_f32 takes may be cut along K into splits (2 .. 8) whose sums, splits * M * N floats, part holds; else null, 1.
extern "C" int locus_gemm_simt(const void* x, int x_dt, const void* w, const void* w2, int w_dt,
                               const void* bias, int bias_dt, void* out, int out_dt,
                               int flags, float act_param, float act_scale, const float* row_scale, const int* scale_rows,
                               const int* x_rows,
                               int x_row_div, int M, int N, int K, long long ldx, long long ldo,
                               const int* tile_expert, const int* tile_row0,
                               const int* tile_rows, const int* n_tiles, int max_tiles,
                               long long w_expert_stride, float* part, int splits, cudaStream_t stream) {
    if (N <= 0 || K <= 0) return LOCUS_ERR_UNSUPPORTED;
    const int accumulate = flags & 1, act = (flags >> 1) & 7;
    if ((act == 1 && w2 != nullptr) || ((act == 2 || act == 4) && w2 == nullptr) || act > 4 || (act == 3 && (w2 != nullptr || !(act_param > 0.f)))) return LOCUS_ERR_UNSUPPORTED;
    if (accumulate && out_dt != LOCUS_DT_F32) return LOCUS_ERR_UNSUPPORTED;
    if (x_rows != nullptr && x_row_div <= 0) return LOCUS_ERR_UNSUPPORTED;
    GemmArgs a;
    a.x = x; a.w = w; a.w2 = w2; a.bias = bias; a.bias_dt = bias_dt; a.out = out;
    a.out_dt = out_dt; a.accumulate = accumulate; a.act = act; a.act_param = act_param; a.act_scale = act_scale; a.row_scale = row_scale; a.scale_rows = scale_rows; a.x_rows = x_rows;
    a.x_row_div = x_row_div; a.M = M; a.N = N; a.K = K; a.ldx = ldx; a.ldo = ldo;
    a.tile_expert = tile_expert; a.tile_row0 = tile_row0; a.tile_rows = tile_rows;
    a.n_tiles = n_tiles; a.w_expert_stride = w_expert_stride; a.part = splits > 1 ? part : nullptr; a.splits = splits > 1 ? splits : 1;
    const int tiles = tile_expert ? max_tiles : ceil_div(M, BM);
    const bool swiglu = w2 != nullptr;
    static_assert(FM == BM, "the grouped tile lists serve both kernels");
    static int n_sm = 0;
    if (n_sm == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n_sm <= 0) {
            n_sm = 0;
            return static_cast<int>(cudaGetLastError());
        }
    }
    // Short sums stay on gemm_simt, whose blocks start and end quicker: up to 32 columns, and one weight's up to 127 while its tiles
    // fit the GPU at once (gemm_simt / gemm_f32: 2,048 x 6,144 x 16 30 / 54 us, x 32 48 / 54, x 64 78 / 70; 64 x 512 x 64
    // 6.3 / 11.1, x 96 8.5 / 12.8, x 128 10.4 / 9.1 in two parts; pairs of 64 x 512 x 32 9.1 / 9.0, x 64 12.1 / 11.0).
    const bool is_short = splits <= 1 && (K <= 32 || (K < 128 && !swiglu && static_cast<long long>(ceil_div(N, 128)) * tiles <= 2 * n_sm));
    if (x_dt == LOCUS_DT_F32 && w_dt == LOCUS_DT_F32 && !is_short && ((K | ldx) & 3) == 0 &&
        ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(w2)) & 15) == 0) {
        if (splits > 1 && (part == nullptr || splits > 8 || swiglu || tile_expert != nullptr || M > 65535)) return LOCUS_ERR_UNSUPPORTED;
        // tiles of 64 weight rows where tiles of 128 would leave SMs without one
        const long long wide = static_cast<long long>(ceil_div(N, swiglu ? 64 : 128)) * tiles * a.splits;
        return wide < n_sm ? launch_f32<8>(a, tiles, swiglu, stream) : launch_f32<16>(a, tiles, swiglu, stream);
    }
    if (splits > 1) return LOCUS_ERR_UNSUPPORTED;
    if (x_dt == LOCUS_DT_F32 && w_dt == LOCUS_DT_F32) return launch<float, float>(a, tiles, swiglu, stream);
    if (x_dt == LOCUS_DT_BF16 && w_dt == LOCUS_DT_BF16) return launch<bf16, bf16>(a, tiles, swiglu, stream);
    if (x_dt == LOCUS_DT_BF16 && w_dt == LOCUS_DT_F32) return launch<bf16, float>(a, tiles, swiglu, stream);
    if (x_dt == LOCUS_DT_F32 && w_dt == LOCUS_DT_BF16) return launch<float, bf16>(a, tiles, swiglu, stream);
    return LOCUS_ERR_UNSUPPORTED;
}
