// Shared by the recurrences that walk a sequence's tokens in blocks of four (delta_rule.cu, wkv.cu).
#pragma once
#include "common.cuh"

// Two float32 at once: each half rounded as the single instruction rounds it.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}

// The sequence that comes `place`-th when the step's are ordered from the longest to the shortest; whole warps call it, up
// to 64 sequences.
#define SEQUENCE_PLACE_MAX 64
__device__ __forceinline__ int sequence_place(const int *seq_start, int n_seqs, int place) {
    const int lane = threadIdx.x & 31;
    const int a = lane < n_seqs ? seq_start[lane + 1] - seq_start[lane] : -1;
    const int b = lane + 32 < n_seqs ? seq_start[lane + 33] - seq_start[lane + 32] : -1;
    int before_a = 0, before_b = 0;  // how many come before this lane's two
    for (int j = 0; j < n_seqs; j++) {
        const int other = __shfl_sync(0xffffffffu, j < 32 ? a : b, j & 31);
        before_a += other > a || (other == a && j < lane), before_b += other > b || (other == b && j < lane + 32);
    }
    const unsigned hit_a = __ballot_sync(0xffffffffu, lane < n_seqs && before_a == place);
    const unsigned hit_b = __ballot_sync(0xffffffffu, lane + 32 < n_seqs && before_b == place);
    return hit_a ? __ffs(hit_a) - 1 : 31 + __ffs(hit_b);
}
