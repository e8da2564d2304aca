// Asynchronous copies into shared memory and pairs of float32 multiply-adds, for all float32 kernels (gla.cu, delta_rule.cu, gemv.cu,
// gemm_simt.cu, attention_f32.cu); sums of several values over a warp (the first three); and how the kernels that walk a
// request's tokens in order (gla.cu, delta_rule.cu) lay a head's state over their warps:
//
// A warp holds two columns of a head's state; lane l keeps of both the rows 128 j + 4 l + {0, 1, 2, 3} (heads of up to 64 rows:
// 2 l + {0, 1}).  A load of 16 bytes a lane from shared memory takes four passes over the banks whether or not lanes read the
// same addresses, so a loaded row has to serve as many columns as possible, and against that stand the lanes that a sum
// crosses and the warps that hide a walk's chain from each other.  Measured for gla_walk at 2,048 tokens of 16 heads of
// 128 x 128: one column to a lane and 8 row groups 310 us with one warp a scheduler, 229 us with the rows shared by four
// warps (bound by the passes); four columns to a lane, one warp a scheduler, 332 us (bound by the chain: 3.3 cycles an
// instruction); two columns, two warps a scheduler, the next token's operands in
// registers: 259 us (for eight such requests 1,390 us, 1,290 with three blocks an SM; the rows shared by two warps: 257 and 1,756 us).
#pragma once

#define WALK_CW 2      // columns of a warp
#define WALK_WARPS 8   // warps of a block: 16 columns of a head; 16 heads of 128 columns are 128 blocks on 148 SMs

// Which kernel takes a request of how many tokens.  A tile costs a block of a walk nearly the same for one token as for 16 (copies,
// barriers, the sums of pairs), a single token a block of the tokens kernels about 0.5 us, of which an SM hides several blocks'.
// 16 heads of 128, token by token / in tiles, gated linear attention and the delta rule: 1 request of 8 tokens 5.6 / 6.4 and
// 5.8 / 6.6 us, of 12 7.6 / 6.8 and 8.4 / 7.2; 8 requests of 16 23 / 31 and 26 / 34, of 24 33 / 37 and 37 / 45, of 32 42 / 40 and 48 / 50;
// 64 requests of 24 242 / 269 and 314 / 325.  Heads of 64, 1 request of 6 tokens 4.9 / 5.1 and 5.1 / 5.0, of 8 5.7 / 5.2 and 6.2 / 4.9.
static inline bool walk_not_needed(int n_rows, int n_seg, int d) {
    return n_rows <= 2LL * n_seg || n_rows <= (d > 64 ? 8 : 6);
}
// Steps of fewer than 64 tokens a request on average, of several requests: the instances that look at every request's length,
// which cost long portions 1 to 2 % (8 requests of 2,048 1,287 -> 1,308 us) and save a walk of tiles for every single token.
static inline bool walk_may_be_mixed(int n_rows, int n_seg) { return n_seg > 1 && n_rows < 64LL * n_seg; }
// The most tokens that such a step takes one by one, by 256 threads for the columns of two blocks.  blocks: 16 columns of a
// head of a request each; more than three an SM hide each other's chains.
static inline int walk_few(long long blocks) { return blocks <= 3 * 148 ? 4 : 20; }

// N bytes (16 or 4) from global to shared memory; `live` false writes zeros and reads nothing.
template <int N>
__device__ __forceinline__ void walk_copy(void* dst, const void* src, bool live) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    const int n = live ? N : 0;
    if constexpr (N == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void walk_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void walk_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

typedef unsigned long long f2;   // two float32 in one register pair

__device__ __forceinline__ f2 f2_pack(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_unpack(f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// v[0 .. N - 1] (N 8, 16 or 32): values to be summed over the warp.  Half of the values change hands at every step until each
// lane has one: 31 exchanges for 32 values instead of 160.  Returns the sum of value walk_sum_index<N>(lane).
template <int N>
__device__ __forceinline__ int walk_sum_index(int lane) {
    return static_cast<int>(__brev(lane & (N - 1)) >> (N == 32 ? 27 : N == 16 ? 28 : 29));
}
template <int N, int MASK = 1>
__device__ __forceinline__ float walk_sum(const float* v, int lane) {
    if constexpr (N == 1) {
        float s = v[0];
#pragma unroll
        for (int m = MASK; m < 32; m <<= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
        return s;
    } else {
        float w[N / 2];
        const bool upper = lane & MASK;
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
            const float send = upper ? v[i] : v[i + N / 2], keep = upper ? v[i + N / 2] : v[i];
            w[i] = keep + __shfl_xor_sync(0xffffffffu, send, MASK);
        }
        return walk_sum<N / 2, MASK * 2>(w, lane);
    }
}
