// What the kernels that walk a request's tokens in order share (gla.cu, delta_rule.cu): asynchronous copies of the next
// tokens' operands into shared memory, pairs of float32 multiply-adds, and sums over the row groups of a warp.
//
// A warp holds two columns of a head's state; lane l keeps of both the rows 128 j + 4 l + {0, 1, 2, 3} (heads of up to 64 rows:
// 2 l + {0, 1}).  A load of 16 bytes a lane from shared memory takes four passes over the banks whether or not lanes read the
// same addresses, so a loaded row has to serve as many columns as possible, and against that stand the lanes that a sum
// crosses and the warps that hide a walk's chain from each other.  Measured for gla_walk at 2,048 tokens of 16 heads of
// 128 x 128: one column to a lane and 8 row groups 310 us with one warp a scheduler, 229 us with the rows shared by four
// warps (bound by the passes); four columns to a lane, one warp a scheduler, 332 us (bound by the chain: 3.3 cycles an
// instruction); two columns, two warps a scheduler, the next token's operands in
// registers: 259 us (for eight such requests 1,390 us; the rows shared by two warps: 257 and 1,756 us).
#pragma once

#define WALK_CW 2      // columns of a warp
#define WALK_WARPS 8   // warps of a block: 16 columns of a head; 16 heads of 128 columns are 128 blocks on 148 SMs

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
