// sl_f32x2.cuh -- packed FP32 arithmetic: two numbers in a register pair, one
// issue slot for both, each half the IEEE operation.
#pragma once
#include <cuda_runtime.h>

namespace sl {
namespace f2 {

typedef unsigned long long F32x2;

__device__ __forceinline__ F32x2 pair2(float a, float b)
{
    F32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 split2(F32x2 v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ F32x2 add2(F32x2 a, F32x2 b)
{
    F32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F32x2 mul2(F32x2 a, F32x2 b)
{
    F32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F32x2 fma2(F32x2 a, F32x2 b, F32x2 c)
{
    F32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

}  // namespace f2
}  // namespace sl
