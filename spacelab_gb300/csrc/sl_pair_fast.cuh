// sl_pair_fast.cuh -- the non-contact pair force of the exact form with every
// operation after the geometry rounded in unpacked integer arithmetic.
//
// The reference's force (ColliderSingleCore.cpp:104-227, 249-250) past |r|^2
// is a chain of IEEE multiplications and divisions.  Here a value is a Sig: a
// 64-bit significand m with its top bit set and, once rounded, its low 11
// bits zero (53 significant bits), and an exponent e, value m 2^(e - 63).
// Each operation forms the exact result's leading 64 bits to within a few
// units and rounds to nearest at bit 11 (round53).  Nothing is packed back
// into a double between the operations and nothing branches: where the
// dropped bits lie so near the midpoint that the estimate's error could
// decide, or a value leaves a wide exponent range, a flag is raised and the
// caller evaluates the whole pair again by the general routine
// (sl_tile_exact.cuh), whose results hold for all operands.  About 4% of the
// pairs are flagged.  An unflagged result is the IEEE round-to-nearest-even
// one, bit for bit.
//
// The errors of the estimates, in units of bit 0 before normalisation (a left
// shift of one doubles them); the truncation of mulhi is (-1, 0]:
//   root_sig    Y - 2^64 / sqrt(f) in (-3, 2): the residual e2 carries the
//               two truncations centred, [-1, 1), times Y 2^-63 <= 2, and the
//               product's own truncation; H = F Y 2^-64 in (-3, 1), since
//               F Y 2^-127 < 1, and in (-6, 2) once doubled
//   its reciprocal  Yd - 2^127 / m_d in (-2, 1): the residual to a half either
//               way, times 2^64 / m_d <= 2, and a truncation;
//               r_k / d = m_r Yd 2^-64 in (-3, 1)
//   recip_sig64 R - 2^127 / m in (-1, 2): the residual's truncation [0, 1)
//               times 2^64 / m <= 2, and a truncation;
//               num / den = m_n R 2^-64 in (-2, 2)
//   F / mass    rm in (-1, 0], m_F rm 2^-64 in (-2, 0]
//   product     m_a m_b 2^-64 in (-1, 0]
// tests/test_pair_fast.py measures the reciprocals' errors exactly and
// compares unflagged results with IEEE double operations, on the host.
#pragma once
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define SL_PF_FN __host__ __device__ __forceinline__
#else
#include <cmath>
#define SL_PF_FN inline
#endif

namespace sl {
namespace pf {

typedef unsigned long long u64;

SL_PF_FN u64 mulhi(u64 a, u64 b)
{
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (u64)(((unsigned __int128)a * b) >> 64);
#endif
}

SL_PF_FN u64 bits_of(double x)
{
#ifdef __CUDA_ARCH__
    return (u64)__double_as_longlong(x);
#else
    u64 u;
    std::memcpy(&u, &x, 8);
    return u;
#endif
}

SL_PF_FN double from_bits(u64 u)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double x;
    std::memcpy(&x, &u, 8);
    return x;
#endif
}

// Hardware seeds (relative error below 2^-22): on the host a float operation
// with an error of the same size, so that the bounds are exercised.
#ifndef __CUDA_ARCH__
inline float& host_seed_error()
{
    static float e = 0.0f;  // relative error put on the host's seeds
    return e;
}
#endif

SL_PF_FN uint32_t rsqrt_seed(uint32_t f_bits)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(f_bits)));
    return __float_as_uint(y);
#else
    float f;
    std::memcpy(&f, &f_bits, 4);
    const float y = (float)((1.0 / std::sqrt((double)f)) * (1.0 + host_seed_error()));
    uint32_t u;
    std::memcpy(&u, &y, 4);
    return u;
#endif
}

SL_PF_FN uint32_t rcp_seed(uint32_t g_bits)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(g_bits)));
    return __float_as_uint(y);
#else
    float g;
    std::memcpy(&g, &g_bits, 4);
    const float y = (float)((1.0 / (double)g) * (1.0 + host_seed_error()));
    uint32_t u;
    std::memcpy(&u, &y, 4);
    return u;
#endif
}

struct Sig {
    u64 m;
    int e;
};

// What the operations of one pair found: `near` is the least distance (plus
// kNear - width) of a result's dropped bits into its midpoint window, `top`
// the AND of the significands' high words (top bit clear: one of them left
// its range), `range` nonzero where an exponent left its range.
constexpr uint32_t kNear = 31;
struct Flags {
    uint32_t near = 0xffffu, top = 0xffffffffu, range = 0;
    SL_PF_FN bool sure() const { return near > kNear && (top >> 31) != 0 && range == 0; }
};

// a nonzero normal double's magnitude; others give e = -1023 or 1024, which
// the callers' range checks refuse
SL_PF_FN Sig unpack(double x)
{
    const u64 b = bits_of(x);
    return {(b << 11) | 0x8000000000000000ull, (int)((uint32_t)(b >> 52) & 0x7ffu) - 1023};
}

SL_PF_FN double pack(const Sig& s, uint32_t sign)  // sign: 0 or 0x80000000
{
    const u64 v = s.m >> 11;  // hidden bit at 52
    const uint32_t hi = ((uint32_t)(v >> 32) + ((uint32_t)(s.e + 1022) << 20)) | sign;
    return from_bits(((u64)hi << 32) | (uint32_t)v);
}

// e outside [-(BITS/2 - 1), BITS/2] raises the flag
template <uint32_t SPAN>
SL_PF_FN void check_range(Flags& fl, int e)
{
    fl.range |= (uint32_t)(e + (int)(SPAN / 2 - 1)) & ~(SPAN - 1);
}

// Whether two coordinates are equal up to their signs (zeros of both signs are)
SL_PF_FN bool equal(double x, double y) { return ((bits_of(x) ^ bits_of(y)) << 1) == 0; }

// An estimate H in [2^62, 2^64) of value H 2^(e - 63), normalised and rounded
// to nearest at bit 11.  The exact value lies in (H - BELOW, H + ABOVE) after
// normalisation, so only dropped bits in [1024 - ABOVE, 1024 + BELOW] leave
// the direction open.
template <uint32_t ABOVE, uint32_t BELOW>
SL_PF_FN Sig round53(u64 H, int e, Flags& fl)
{
    static_assert(ABOVE + BELOW <= kNear, "window");
    const uint32_t c = (uint32_t)(H >> 63) ^ 1u;
    H <<= c;
    const u64 M = H + 1024;
    const uint32_t t = (((uint32_t)M + ABOVE) & 2047u) + (kNear - ABOVE - BELOW);
    fl.near = t < fl.near ? t : fl.near;
    fl.top &= (uint32_t)(M >> 32);
    return {M & ~2047ull, e - (int)c};
}

// RN(a b): the exact product lies in [H, H + 1), [H, H + 2) once shifted by
// one (H then even), so the open case is the midpoint's own bits alone.
SL_PF_FN Sig mul(const Sig& a, const Sig& b, Flags& fl) { return round53<0, 0>(mulhi(a.m, b.m), a.e + b.e + 1, fl); }

// RN(a / b) for r = recip_sig of b's 53-bit significand (floor of 2^127 / m_b
// to within one unit below).
SL_PF_FN Sig div_fixed(const Sig& a, u64 r, int eb, Flags& fl)
{
    return round53<3, 0>(mulhi(a.m, r), a.e - eb, fl);
}

// RN(a / d) for r = recip_of_root's estimate of 2^127 / m_d.
SL_PF_FN Sig div_root(const Sig& a, u64 r, int ed, Flags& fl) { return round53<6, 2>(mulhi(a.m, r), a.e - ed, fl); }

// 2^127 / m to within (-1, 2): a seed and two Newton steps r <- r + r (1 - g r),
// g = m 2^-63.  The first step takes the residual's top 32 bits, the second
// the residual whole (it is below 2^20), times the top 32 bits of r.
SL_PF_FN u64 recip_sig64(u64 m, Flags& fl)
{
    const uint32_t sb = rcp_seed(0x3f800000u | ((uint32_t)(m >> 40) & 0x7fffffu));
    uint32_t s = sb - 0x3e800000u;  // r0 2^24 for r0 in [1/2, 1]
    s = s > 0xffffffu ? 0xffffffu : s;
    const u64 R0 = (u64)s << 40;
    const long long e1 = (long long)(0x8000000000000000ull - mulhi(m, R0));  // (1 - g r0) 2^63, below 2^42
    // r0 lies below 1/g after the step; the 2^14 keeps it so through the truncations
    const u64 R1 = R0 + (u64)(((long long)(int32_t)s * (int32_t)(e1 >> 11)) >> 12) - 0x4000ull;
    const uint32_t e2 = (uint32_t)(0x8000000000000000ull - mulhi(m, R1));
    const u64 R = R1 + (((R1 >> 32) * (u64)e2) >> 31);
    fl.top &= (uint32_t)(R >> 32);
    return R;
}

// |r|^2 -> d = RN(sqrt(d2)) and 2^127 / m_d, without the square root's exact
// remainder: f = d2 2^(-2p) in [1, 4), F = f 2^62, Y ~ 2^64 / sqrt(f) by a
// seed and two Newton steps y <- y + y (1 - f y^2) / 2, H = F Y 2^-64 ~
// sqrt(f) 2^62.  The reciprocal of the rounded root is Y moved by the
// rounding (first order) and corrected by its own residual.
struct Root {
    Sig d;
    u64 rec;
};

SL_PF_FN Root root_sig(double d2, Flags& fl)
{
    const u64 b = bits_of(d2);
    const int E = (int)((uint32_t)(b >> 52)) - 1023;  // d2 > 0 and normal
    const uint32_t odd = (uint32_t)E & 1u;
    const int p = E >> 1;
    const u64 M2 = (b << 11) | 0x8000000000000000ull;
    const u64 F = M2 >> (1 - odd);
    const uint32_t sb = rsqrt_seed(((127u + odd) << 23) | ((uint32_t)(M2 >> 40) & 0x7fffffu));
    uint32_t s = sb - 0x3e800000u;  // y0 2^24 for y0 in [1/2, 1]
    s = s > 0xffffffu ? 0xffffffu : s;
    const long long e1 = (long long)(0x2000000000000000ull - mulhi(((u64)s * s) << 15, F));  // (1 - f y0^2) 2^61
    const u64 Y1 = ((u64)s << 40) + (u64)(((long long)(int32_t)s * (int32_t)(e1 >> 10)) >> 12) - 0x4000ull;
    const uint32_t e2 = (uint32_t)(0x3fffffffffffffffull - mulhi(mulhi(Y1, Y1), F));  // (1 - f y1^2) 2^62, >= 0
    const u64 Y = Y1 + (((Y1 >> 32) * (u64)e2) >> 31);
    fl.top &= (uint32_t)(Y >> 32);
    const u64 H = mulhi(F, Y) << 1;
    const Sig d = round53<6, 2>(H, p, fl);
    // 2^127 / (m + e) = Y - e Y^2 2^-127 for d's significand m + e, m ~ H
    const int e = (int)((uint32_t)d.m - (uint32_t)H);
    const uint32_t yh = (uint32_t)(Y >> 32);
    const uint32_t qh = (uint32_t)(((u64)yh * yh) >> 32);
    const u64 Yd0 = Y - (u64)(long long)((e * (int)(qh >> 14)) >> 17);
    // its residual 2^63 - m_d Yd0 2^-64 is a few units; centred by a half
    const int D = (int)(uint32_t)(0x8000000000000000ull - mulhi(d.m, Yd0));
    const u64 Yd = Yd0 + (u64)(long long)(((2 * D - 1) * (int)(yh >> 16)) >> 16);
    fl.top &= (uint32_t)(Yd >> 32);
    return {d, Yd};
}

// P num / (S S T T), the vdW coefficient (ColliderSingleCore.cpp:221-225):
// every product and the quotient rounded.  num must be a normal number with
// an exponent in +-500.
SL_PF_FN Sig vdw_coef(const Sig& P, double num, double S, double T, Flags& fl)
{
    const Sig s = unpack(S), t = unpack(T), u = unpack(num);
    check_range<256>(fl, s.e);
    check_range<256>(fl, t.e);
    const Sig den = mul(mul(mul(s, s, fl), t, fl), t, fl);
    const Sig q = round53<4, 4>(mulhi(u.m, recip_sig64(den.m, fl)), u.e - den.e, fl);
    const Sig c = mul(P, q, fl);
    check_range<1024>(fl, c.e);
    return c;
}

// The per-sphere operands of a pair.  Exponents in range: R in +-120, the
// mass in +-200 (for `rm`, its recip_sig), cR3 in +-500 -- the caller checks
// them once per sphere (in_range).
struct Sphere {
    double R;
    Sig sR;             // unpacked R
    double cR3;         // A only: ((Ha/6 64) R) R R
    u64 rm;
    int em;
};

SL_PF_FN bool in_range(const Sphere& p)
{
    const int er = unpack(p.R).e;
    return er > -120 && er < 120 && p.em > -200 && p.em < 200;
}
SL_PF_FN bool is_zero(double x) { return (bits_of(x) << 1) == 0; }
SL_PF_FN bool in_range_cR3(double cR3)
{
    const int e = unpack(cR3).e;
    return e > -500 && e < 500;
}

// What is the same for every pair of a tile whose spheres all have one
// radius and one mass.
struct Uniform {
    double sum, c4;  // R + R, (4 R) R
    Sig P;           // ((cR3 R) R) R
};

struct Pair {
    double overlap, h;
    double ta[3], tb[3];  // F / m[A], -(F / m[B])
    Flags fl;
};

// The pair (A, B) out of contact, r = pos[B] - pos[A]
// (ColliderSingleCore.cpp:104-227, 249-250).  The FP64 pipe keeps the adds;
// the products are formed here and packed where an add follows.  On GB300 a
// warp's FP64 operation holds the SM's unit for 19 cycles and a product here
// takes some 20 instructions of four schedulers: with all of these operations
// on the FP64 pipe it was 95% busy, at 37% of the issue slots.
// overlap is valid whenever `fl` is sure (contact: overlap > 0).
//
// ZEROS: a component of r may be zero (spheres in a plane or on a grid), and cR3
// zero (no cohesion) or negative (repulsion); it is positive otherwise.  A zero's
// square and force are zeros, the force's with its sign; a one takes its place in
// the operations, and says nothing.  Without it a zero component raises the range
// flag.  It costs some thirty instructions a pair, so the tiles take it only where
// they meet such pairs.
template <bool UNI, bool ZEROS = false>
SL_PF_FN Pair pair_terms(double rx, double ry, double rz, const Sphere& A, const Sphere& B, const Uniform& u,
                         long long h_min_bits)
{
    Pair o;
    Flags fl;
    const double r[3] = {rx, ry, rz};
    const Sig one{0x8000000000000000ull, 0};
    const bool none = ZEROS && is_zero(A.cR3);
    Sig sr[3];
    double sq[3];
    bool zero[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        zero[c] = ZEROS && is_zero(r[c]);
        sr[c] = zero[c] ? one : unpack(r[c]);
        check_range<256>(fl, sr[c].e);
        sq[c] = pack(mul(sr[c], sr[c], fl), 0);
        if (zero[c]) sq[c] = 0.0;
    }
    if (ZEROS && zero[0] && zero[1] && zero[2]) fl.range = 1;
    const Root root = root_sig(sq[0] + sq[1] + sq[2], fl);             // :107
    o.overlap = (UNI ? u.sum : A.R + B.R) - pack(root.d, 0);           // :104, :110
    u64 hb = bits_of(o.overlap) & 0x7fffffffffffffffull;               // :211-215
    if ((long long)hb < h_min_bits) hb = (u64)h_min_bits;
    o.h = from_bits(hb);
    const Sig sh = unpack(o.h);
    check_range<512>(fl, sh.e);
    const double h2 = pack(mul(sh, sh, fl), 0);
    const double tb = pack(mul(Sig{B.sR.m, B.sR.e + 1}, sh, fl), 0);  // (2 R[B]) h
    double S, T;
    Sig P = none ? one : u.P;
    if (UNI) {
        S = h2 + tb + tb;
        T = S + u.c4;
    } else {
        S = h2 + pack(mul(Sig{A.sR.m, A.sR.e + 1}, sh, fl), 0) + tb;
        T = S + pack(mul(Sig{A.sR.m, A.sR.e + 2}, B.sR, fl), 0);
        P = mul(mul(mul(none ? one : unpack(A.cR3), B.sR, fl), B.sR, fl), B.sR, fl);
    }
    const Sig coef = vdw_coef(P, o.h + A.R + B.R, S, T, fl);           // :221-225
    // the significands hold magnitudes: a negative cR3 turns the signs
    const uint32_t csign = ZEROS ? (uint32_t)(bits_of(A.cR3) >> 32) & 0x80000000u : 0u;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const uint32_t sign = ((uint32_t)(bits_of(r[c]) >> 32) & 0x80000000u) ^ csign;
        // alone beside two zeros: RN(sqrt(RN(x x))) = |x|, a quotient of one
        const bool unit = ZEROS && (zero[c] || (zero[(c + 1) % 3] && zero[(c + 2) % 3]));
        const Sig n = unit ? one : div_root(sr[c], root.rec, root.d.e, fl);
        const Sig F = mul(coef, n, fl);                                // :227
        const bool nil = none || zero[c];
        o.ta[c] = nil ? from_bits((u64)sign << 32) : pack(div_fixed(F, A.rm, A.em, fl), sign);  // :249
        // -(F/m[B]), :250; equal masses: RN(-x) = -RN(x)
        o.tb[c] = UNI || nil ? from_bits(bits_of(o.ta[c]) ^ 0x8000000000000000ull)
                             : pack(div_fixed(F, B.rm, B.em, fl), sign ^ 0x80000000u);
    }
    o.fl = fl;
    return o;
}

}  // namespace pf
}  // namespace sl
