// sl_parts.cuh -- FP64 positions as three FP32 parts whose pair differences
// come out as if subtracted in FP64 and rounded to FP32 once (the
// FP64-accumulating mixed form's r = pos[B] - pos[A]).
//
// a1 = the float nearest a; a2 = the rest rounded to a multiple of
// 2^-23 ulp(a1), at most half an ulp(a1) (grid_part); a3 = what is left.  Then,
// for two numbers,
//   - a1 - b1 with its error is exact (TwoSum);
//   - a2 - b2 is exact where a1 and b1 lie within a factor of four of each
//     other (multiples of the finer grid below 2^24 of it); elsewhere it is
//     rounded at 2^-24 of an ulp of the larger, some 2^-22 ulp of the difference;
//   - the sum of the two with its error is exact (Fast2Sum): the first is zero,
//     or the larger, or a multiple of the sum's last place.
// The error terms and a3 - b3 are below 2^-22 of the result or it is their
// exact sum.  tests/test_parts.py measures at most 0.500 ulp on the host, from
// the origin to 1e8 radii away.  With a2 the float nearest the rest and no Fast2Sum
// a component near 2 radii was off by up to 3.75 ulp at 1e4 radii and 44 at 1e6,
// and a small one near the origin by 38, for three additions a component less.
#pragma once
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define SL_PARTS_FN __host__ __device__ __forceinline__
#else
#define SL_PARTS_FN inline
#endif

namespace sl {
namespace parts {

// lo rounded to a multiple of 2^-23 ulp(hi), for |lo| <= ulp(hi) / 2: by adding
// and taking away 1.5 ulp(hi).  Below 2^-79 in the scaled lengths lo stays.
SL_PARTS_FN float grid_part(float hi, float lo)
{
    uint32_t h;
    std::memcpy(&h, &hi, 4);
    const uint32_t e = (h >> 23) & 0xffu;
    if (e < 48) return lo;
    const uint32_t magic = ((e - 23) << 23) | 0x400000u;
    float m;
    std::memcpy(&m, &magic, 4);
    return (lo + m) - m;
}

SL_PARTS_FN float sub3(float a1, float a2, float a3, float b1, float b2, float b3)
{
    const float s = a1 - b1;
    const float bp = s - a1;
    const float e1 = (a1 - (s - bp)) - (b1 + bp);
    const float t = a2 - b2;
    const float q = s + t;
    const float z = t - (q - s);
    return q + ((z + e1) + (a3 - b3));
}

}  // namespace parts
}  // namespace sl
