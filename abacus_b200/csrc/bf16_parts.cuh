// Float32 numbers as sums of three bfloat16 numbers, for products on the tensor cores that give up no digit.
#pragma once
#include <stdint.h>

// Two numbers as three pairs of bfloat16 (the lower half of a word: the first number): 8 + 8 + 8 bits, each rounded to nearest; what is
// left over is below 2^-26 of a number.
__device__ __forceinline__ void split_pair(float a, float b, uint32_t &p1, uint32_t &p2, uint32_t &p3) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p1) : "f"(b), "f"(a));
    a -= __uint_as_float(p1 << 16), b -= __uint_as_float(p1 & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p2) : "f"(b), "f"(a));
    a -= __uint_as_float(p2 << 16), b -= __uint_as_float(p2 & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p3) : "f"(b), "f"(a));
}
