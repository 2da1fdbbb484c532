// sl_df.cuh -- double-float arithmetic: a value held as an unevaluated sum
// hi + lo of two FP32 numbers (|lo| <= ulp(hi)/2), about 48 significant
// bits, built from error-free transformations on the FP32 pipe (Knuth's
// TwoSum, Dekker's Fast2Sum, and the FMA-based TwoProduct).  The mixed form
// uses it where it needs more than FP32: pair displacements, |r|^2, the
// squared gap and the per-sphere sums.  GB300's FP32 pipe is ~72x its FP64
// pipe, so these few FP32 operations cost far less than one FP64 operation.
//
// Every function here must be compiled without reassociation of FP32
// additions (nvcc's default); the FMAs are explicit.
#pragma once
#include <cuda_runtime.h>

#include "sl_f32x2.cuh"

namespace sl {
namespace df {

struct F2 {
    float hi, lo;
};

// s + e == a + b exactly (any a, b without overflow)
__device__ __forceinline__ F2 two_sum(float a, float b)
{
    const float s = a + b;
    const float bp = s - a;
    const float e = (a - (s - bp)) + (b - bp);
    return {s, e};
}

// s + e == a + b exactly when |a| >= |b| (or a == 0)
__device__ __forceinline__ F2 fast_two_sum(float a, float b)
{
    const float s = a + b;
    return {s, b - (s - a)};
}

// p + e == a * b exactly (barring underflow)
__device__ __forceinline__ F2 two_prod(float a, float b)
{
    const float p = a * b;
    return {p, fmaf(a, b, -p)};
}

__device__ __forceinline__ F2 add(F2 a, F2 b)
{
    F2 s = two_sum(a.hi, b.hi);
    s.lo += a.lo + b.lo;
    return fast_two_sum(s.hi, s.lo);
}

__device__ __forceinline__ F2 sub(F2 a, F2 b)
{
    F2 s = two_sum(a.hi, -b.hi);
    s.lo += a.lo - b.lo;
    return fast_two_sum(s.hi, s.lo);
}

__device__ __forceinline__ F2 sqr(F2 a)
{
    F2 p = two_prod(a.hi, a.hi);
    p.lo = fmaf(2.0f * a.hi, a.lo, p.lo);
    return fast_two_sum(p.hi, p.lo);
}

// Running sum of FP32 terms in three parts, a + b + c: the rounding error of
// each addition into a goes exactly into b, and b's into c -- some 70 bits, so
// a sum of 32 terms is closer to the exact one than a running FP64 sum, for
// 13 FP32 additions a term.
struct Sum3 {
    float a, b, c;
    __device__ __forceinline__ void add(float v)
    {
        const F2 t = two_sum(a, v);
        a = t.hi;
        const F2 u = two_sum(b, t.lo);
        b = u.hi;
        c += u.lo;
    }
};

// Two Sum3 at once, in packed arithmetic: the halves are separate sums, each
// with the operations of Sum3.
struct Sum3x2 {
    f2::F32x2 a, b, c;
    __device__ __forceinline__ void add(f2::F32x2 v)
    {
        using namespace f2;
        const F32x2 m1 = pair2(-1.0f, -1.0f);  // x - y = y m1 + x, exactly rounded
        const F32x2 s = add2(a, v);
        const F32x2 vp = fma2(a, m1, s);
        const F32x2 e = add2(fma2(fma2(vp, m1, s), m1, a), fma2(vp, m1, v));
        a = s;
        const F32x2 t = add2(b, e);
        const F32x2 ep = fma2(b, m1, t);
        const F32x2 r = add2(fma2(fma2(ep, m1, t), m1, b), fma2(ep, m1, e));
        b = t;
        c = add2(c, r);
    }
};

// Compensated running sum (Neumaier): s carries the sum, c the exact
// rounding errors of each addition; the value is s + c.
struct Sum {
    float s, c;
    __device__ __forceinline__ void add(float v)
    {
        const F2 t = two_sum(s, v);
        s = t.hi;
        c += t.lo;
    }
};

}  // namespace df
}  // namespace sl
