// Two float32 values an instruction: each half rounds as the scalar instruction does, and takes half an issue slot.
#pragma once
#include "common.cuh"

__device__ __forceinline__ unsigned long long f2_pair(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ unsigned long long f2_twice(float x) { return f2_pair(x, x); }
__device__ __forceinline__ float f2_lo(unsigned long long x) { return __uint_as_float((unsigned)x); }
__device__ __forceinline__ float f2_hi(unsigned long long x) { return __uint_as_float((unsigned)(x >> 32)); }
__device__ __forceinline__ unsigned long long f2_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long f2_add(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long f2_mul(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
