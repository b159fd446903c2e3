// Arithmetic on one point (float) or two (F2), with every rounding explicit.
//
// F2 holds two floats in one 64-bit register: sm_100a adds, multiplies and
// multiply-adds both halves in one instruction, each half rounded as the
// scalar instruction rounds it, so a thread that advances two points spends
// half the issue slots on arithmetic.  vmul, vadd and vmad are the same
// operations for float and F2: code written in them gives the same bits for
// either, because the compiler contracts none of them.  vmad(a, b, c) is
// a * b + c, fused in the default build and rounded twice in the build that
// follows the reference's order (CGFDM_EXACT).
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

__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float vsub(float a, float b) { return __fsub_rn(a, b); }

template <class V>
__device__ __forceinline__ V vmad(V a, V b, V c)
{
#ifdef CGFDM_EXACT
    return vadd(vmul(a, b), c);
#else
    return vfma(a, b, c);
#endif
}

// both halves (or the float itself) the same value
template <class V>
__device__ __forceinline__ V bc(float x);
template <>
__device__ __forceinline__ float bc<float>(float x)
{
    return x;
}
template <>
__device__ __forceinline__ F2 bc<F2>(float x)
{
    return pk(x, x);
}
// half l (0 or 1); a float has half 0 only
__device__ __forceinline__ float half_of(float x, int) { return x; }
__device__ __forceinline__ float half_of(F2 x, int l)
{
    float a, b;
    unpk(x, a, b);
    return l ? b : a;
}

}  // namespace cgfdm
