// Packed FP32 arithmetic: two points in one register pair.
//
// F2 holds two floats in one 64-bit register; sm_100a adds, multiplies and
// multiply-adds both halves in one instruction, each half rounded as the
// scalar instruction rounds it, so a thread that advances two points spends
// half the issue slots on arithmetic.  (A packed constant takes two registers.)
#pragma once

#include <cuda_runtime.h>

namespace cgfdm {

struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 pk(float a, float b)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ F2 pk(float a) { return pk(a, a); }
__device__ __forceinline__ void unpk(F2 x, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
}
__device__ __forceinline__ F2 vadd(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 vmul(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 vfma(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ F2 vsub(F2 a, F2 b) { return vfma(b, pk(-1.0f), a); }   // exact product: one rounding

}  // namespace cgfdm
