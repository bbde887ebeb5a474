// f32x2.cuh -- packed FP32 arithmetic of sm_100 and later: two IEEE FP32 operations per lane and
// instruction (add / sub / mul / fma .rn.f32x2), each half rounded exactly as the scalar
// operation rounds it.  The FP32 pipe takes two cycles for a packed instruction, one for a
// scalar one, so the rate is the same, but the issue slots it leaves free go to the integer
// pipe, the rsqrt unit and shared memory (measured on GB300: 2.25 cycles per packed add, 2.5
// for a packed FMA together with an integer add).
#pragma once

#include <cuda_runtime.h>

namespace redgb {

typedef unsigned long long f2;  // {low, high} FP32

__device__ __forceinline__ f2 f2_pack(float lo, float hi)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}

__device__ __forceinline__ f2 f2_dup(float v) { return f2_pack(v, v); }

__device__ __forceinline__ void f2_unpack(f2 v, float& lo, float& hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

__device__ __forceinline__ f2 f2_add(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ f2 f2_sub(f2 a, f2 b)
{
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ f2 f2_mul(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

}  // namespace redgb
