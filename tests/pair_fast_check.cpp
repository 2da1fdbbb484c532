// Host check of the unpacked integer arithmetic of the exact pair force
// (spacelab_gb300/csrc/sl_pair_fast.cuh): the estimates' errors against exact
// integer arithmetic, and every unflagged result against the host's IEEE
// double operations, over random operands, few-bit ones, operands near a
// power of two or with all-ones significands, exact ties, zeros, subnormals,
// infinities and NaN, with seeds up to 2^-22 off either way.
// Prints "<op> <cases> <flagged> <min error> <max error>" and "mismatches N".
#include "sl_pair_fast.cuh"

#include <cfloat>
#include <cstdio>
#include <cstdlib>
#include <random>

using namespace sl::pf;
typedef unsigned __int128 u128;

static std::mt19937_64 rng(12345);
static unsigned long long bad = 0;

static double operand(int lo, int hi)
{
    const u64 r = rng();
    const int e = lo + (int)(rng() % (unsigned)(hi - lo + 1));
    u64 m = rng() & 0xfffffffffffffull;
    switch (r % 10) {
    case 0: m &= ~0ull << (rng() % 52); break;                  // few bits: exact products and ties
    case 1: m = (1ull << (rng() % 8)) - 1; break;               // just above a power of two
    case 2: m = 0xfffffffffffffull - (rng() % 8); break;        // just below one
    case 3: m &= 0xfffffull << 32; break;                       // 20 leading bits
    default: break;
    }
    return from_bits(((u64)(e + 1023) << 52) | m);
}

struct Range {
    double lo = 0, hi = 0;
    unsigned long long n = 0, flagged = 0;
    void err(double e) { lo = e < lo ? e : lo; hi = e > hi ? e : hi; }
    void print(const char* name) const { std::printf("%s %llu %llu %.3f %.3f\n", name, n, flagged, lo, hi); }
};

static void same(const char* what, double got, double want)
{
    if (bits_of(got) != bits_of(want) && ++bad <= 10) std::printf("mismatch %s: got %a want %a\n", what, got, want);
}


static u64 recip_of(double b)
{
    u64 q = 0, rem = 0;
    const u64 mb = (bits_of(b) & 0xfffffffffffffull) | (1ull << 52);
    for (int bit = 115; bit >= 0; --bit) {
        rem = (rem << 1) | 1ull;
        if (rem >= mb) {
            rem -= mb;
            if (bit < 64) q |= 1ull << bit;
        }
    }
    return q;
}

// R - 2^127 / m in units, exactly: (2^127 - m R) / m
static double recip_err(u64 R, u64 m)
{
    const u128 p = (u128)R * m, one = (u128)1 << 127;
    return p >= one ? (double)(long double)(p - one) / (double)m : -((double)(long double)(one - p) / (double)m);
}

static Range pairs;

// A whole pair in lengths, masses and strengths of any scale, against the
// reference's expressions in IEEE doubles.
template <bool UNI>
static void pair_case(long i)
{
    const int sc = (int)(rng() % 40) - 30, sm = (int)(rng() % 60) - 50;
    const double Ra = operand(sc, sc), Rb = UNI ? Ra : operand(sc - 1, sc + 1);
    const double ma = operand(sm, sm), mb = UNI ? ma : operand(sm - 1, sm + 1);
    const double cR3 = operand(-130, -60), hmin = 0.1 * Ra;
    double r[3];
    for (double& x : r) x = operand(sc - 3, sc + (int)(rng() % 7)) * (rng() & 1 ? 1 : -1);
    const Sphere A{Ra, unpack(Ra), cR3, recip_of(ma), unpack(ma).e}, B{Rb, unpack(Rb), 0.0, recip_of(mb), unpack(mb).e};
    const Uniform un{Ra + Rb, (4 * Ra) * Rb, unpack(cR3 * Rb * Rb * Rb)};
    long long hm;
    std::memcpy(&hm, &hmin, 8);
    const Pair p = pair_terms<UNI>(r[0], r[1], r[2], A, B, un, hm);
    ++pairs.n;
    if (!p.fl.sure()) {
        ++pairs.flagged;
        return;
    }
    const double d = std::sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
    const double overlap = (Ra + Rb) - d;
    same("overlap", p.overlap, overlap);
    double h = std::fabs(overlap);
    if (h < hmin) h = hmin;
    same("h", p.h, h);
    const double S = h * h + (2 * Ra) * h + (2 * Rb) * h, T = S + (4 * Ra) * Rb;
    const double coef = cR3 * Rb * Rb * Rb * ((h + Ra + Rb) / (S * S * T * T));
    for (int c = 0; c < 3; ++c) {
        const double F = coef * (r[c] / d);
        same("F/m[A]", p.ta[c], F / ma);
        same("-F/m[B]", p.tb[c], -(F / mb));
    }
    (void)i;
}

int main(int argc, char** argv)
{
    const long n = argc > 1 ? atol(argv[1]) : 1000000;
    const float off[5] = {0.0f, 2.3e-7f, -2.3e-7f, 1.2e-7f, -1.2e-7f};
    Range rsq, rec, rcp, div, prod, quot;
    for (long i = 0; i < n; ++i) {
        host_seed_error() = off[i % 5];
        {  // square root, reciprocal of the rounded root, three quotients
            const double rx = operand(-20, -3) * (rng() & 1 ? 1 : -1), ry = operand(-20, -3), rz = operand(-20, -3);
            const double d2 = i & 1 ? rx * rx + ry * ry + rz * rz : operand(-60, 10);
            Flags fl;
            const Root r = root_sig(d2, fl);
            ++rsq.n;
            if (!fl.sure()) {
                ++rsq.flagged;
            } else {
                const double d = std::sqrt(d2);
                same("sqrt", pack(r.d, 0), d);
                rec.err(recip_err(r.rec, r.d.m));
                ++rec.n;
                Flags g = fl;
                const double a = i & 1 ? rx : operand(-70, 10);
                const Sig q = div_root(unpack(a), r.rec, r.d.e, g);
                ++quot.n;
                if (g.sure())
                    same("a/root", pack(q, a < 0 ? 0x80000000u : 0u), a / d);
                else
                    ++quot.flagged;
            }
            if ((fl.top >> 31) && !fl.range) {
                // H against sqrt(f) 2^63 from below and above: H^2 against F' 2^64
                const long double root = sqrtl((long double)d2);
                int ex;
                const long double fr = frexpl(root, &ex);  // [1/2, 1)
                if (ex - 1 == r.d.e) rsq.err((double)((long double)r.d.m - fr * 18446744073709551616.0L) / 1024);
            }
        }
        {  // reciprocal and division
            const double b = operand(-40, 40), a = operand(-40, 40);
            Flags fl;
            const Sig sb = unpack(b), sa = unpack(a);
            const u64 R = recip_sig64(sb.m, fl);
            ++rcp.n;
            if ((fl.top >> 31)) rcp.err(recip_err(R, sb.m));
            const Sig q = round53<4, 4>(mulhi(sa.m, R), sa.e - sb.e, fl);
            if (fl.sure())
                same("a/b", pack(q, 0), a / b);
            else
                ++rcp.flagged;
            // the mass division: the reciprocal made at upload
            const u64 fix = recip_of(b);
            Flags g;
            const Sig dq = div_fixed(sa, fix, sb.e, g);
            ++div.n;
            div.err(recip_err(fix, sb.m));
            if (g.sure())
                same("a/m", pack(dq, 0x80000000u), -(a / b));
            else
                ++div.flagged;
        }
        {  // products
            const double a = operand(-60, 60), b = operand(-60, 60);
            Flags fl;
            const Sig p = mul(unpack(a), unpack(b), fl);
            ++prod.n;
            if (fl.sure())
                same("a*b", pack(p, 0), a * b);
            else
                ++prod.flagged;
        }
        if (i & 1)
            pair_case<false>(i);
        else
            pair_case<true>(i);
    }
    // operands outside the normal range, or far from 1, are flagged
    host_seed_error() = 0.0f;
    const double special[] = {0.0, -0.0, 5e-324, 1e-310, DBL_MIN / 2, DBL_MIN, INFINITY, NAN, DBL_MAX, 1e300, 1e-300};
    const Sphere one{1.0, unpack(1.0), 1e-20, recip_of(1.0), 0};
    for (double x : special) {
        long long hmin;
        const double hm = 0.1;
        std::memcpy(&hmin, &hm, 8);
        const Uniform un{2.0, 4.0, unpack(1e-20)};
        for (int k = 0; k < 3; ++k) {
            const double r[3] = {k == 0 ? x : 3.0, k == 1 ? x : 3.1, k == 2 ? x : -3.2};
            if (pair_terms<true>(r[0], r[1], r[2], one, one, un, hmin).fl.sure() ||
                pair_terms<false>(r[0], r[1], r[2], one, one, un, hmin).fl.sure()) {
                ++bad;
                std::printf("special operand %a accepted\n", x);
            }
        }
        const Sphere odd{x, unpack(x), x, recip_of(1.0), unpack(x).e};
        if (in_range(odd) || in_range_cR3(x)) {
            ++bad;
            std::printf("special constant %a accepted\n", x);
        }
    }
    rsq.print("root");
    rec.print("recip_root");
    quot.print("quotient_root");
    rcp.print("recip");
    div.print("mass_recip");
    prod.print("product");
    pairs.print("pairs");
    std::printf("mismatches %llu\n", bad);
    return bad != 0;
}
