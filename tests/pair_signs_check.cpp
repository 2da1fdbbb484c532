// Host check of the exact pair force's integer path (sl_pair_fast.cuh) in its
// ZEROS form: vdW coefficients of both signs and zero, and zero displacement
// components.  Unflagged results against the reference's expressions in IEEE
// doubles, signs of zeros too.  Prints "<case> <cases> <flagged>" and
// "mismatches N".
#include "sl_pair_fast.cuh"

#include <cstdio>
#include <cstdlib>
#include <random>

using namespace sl::pf;

static std::mt19937_64 rng(777);
static unsigned long long bad = 0;

// a normal number of either sign, exponent lo .. hi
static double number(int lo, int hi, bool neg)
{
    const int e = lo + (int)(rng() % (unsigned)(hi - lo + 1));
    return from_bits(((u64)neg << 63) | ((u64)(e + 1023) << 52) | (rng() & 0xfffffffffffffull));
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

static void same(const char* what, double got, double want)
{
    if (bits_of(got) != bits_of(want) && ++bad <= 10) std::printf("mismatch %s: got %a want %a\n", what, got, want);
}

// One pair against the reference's force (ColliderSingleCore.cpp:104-227,
// 249-250); true if the path settled it.
template <class Terms>
static bool check(Terms terms, const double r[3], double Ra, double Rb, double ma, double mb, double cR3)
{
    const double hmin = 0.1 * Ra;
    long long hm;
    std::memcpy(&hm, &hmin, 8);
    // as in the tiles: with one radius, A's constants are B's
    const Sphere A{Ra, unpack(Ra), cR3, recip_of(ma), unpack(ma).e}, B{Rb, unpack(Rb), cR3, recip_of(mb), unpack(mb).e};
    const Uniform un{Ra + Rb, (4 * Ra) * Rb, unpack(cR3 * Rb * Rb * Rb)};
    const Pair p = terms(r, A, B, un, hm);
    if (!p.fl.sure()) return false;
    const double d = std::sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
    same("overlap", p.overlap, (Ra + Rb) - d);
    double h = std::fabs((Ra + Rb) - d);
    if (h < hmin) h = hmin;
    const double S = h * h + (2 * Ra) * h + (2 * Rb) * h, T = S + (4 * Ra) * Rb;
    const double coef = cR3 * Rb * Rb * Rb * ((h + Ra + Rb) / (S * S * T * T));
    for (int c = 0; c < 3; ++c) {
        const double F = coef * (r[c] / d);
        same("F/m[A]", p.ta[c], F / ma);
        same("-F/m[B]", p.tb[c], -(F / mb));
    }
    return true;
}

struct Count {
    unsigned long long n = 0, flagged = 0;
    void add(bool settled) { ++n, flagged += !settled; }
    void print(const char* name) const { std::printf("%s %llu %llu\n", name, n, flagged); }
};

template <bool UNI>
static Pair zeros(const double r[3], const Sphere& A, const Sphere& B, const Uniform& un, long long hm)
{
    return pair_terms<UNI, true>(r[0], r[1], r[2], A, B, un, hm);
}

int main(int argc, char** argv)
{
    const long n = argc > 1 ? atol(argv[1]) : 100000;
    Count repulsion, plane, line, no_cohesion;
    for (long i = 0; i < n; ++i) {
        const bool uni = i & 1;
        const int sc = (int)(rng() % 20) - 20;
        const double Ra = number(sc, sc, false), Rb = uni ? Ra : number(sc - 1, sc + 1, false);
        const double ma = number(-40, -38, false), mb = uni ? ma : number(-40, -38, false);
        double r[3];
        for (double& x : r) x = number(sc + 1, sc + 6, rng() & 1);
        const auto care = [&](const double* d, double cR3) {
            return uni ? check(zeros<true>, d, Ra, Rb, ma, mb, cR3) : check(zeros<false>, d, Ra, Rb, ma, mb, cR3);
        };
        repulsion.add(care(r, number(-100, -70, true)));
        const double nil = rng() & 1 ? 0.0 : -0.0;
        no_cohesion.add(care(r, nil));
        const int c = (int)(rng() % 3);
        r[c] = rng() & 1 ? 0.0 : -0.0;
        plane.add(care(r, number(-100, -70, rng() & 1)));
        no_cohesion.add(care(r, nil));
        r[(c + 1) % 3] = rng() & 1 ? 0.0 : -0.0;
        line.add(care(r, number(-100, -70, rng() & 1)));
        r[(c + 2) % 3] = rng() & 1 ? 0.0 : -0.0;
        if (care(r, number(-100, -70, false))) {  // two centres in one place
            ++bad;
            std::printf("zero distance accepted\n");
        }
    }
    repulsion.print("repulsion");
    plane.print("plane");
    line.print("line");
    no_cohesion.print("no_cohesion");
    std::printf("mismatches %llu\n", bad);
    return bad != 0;
}
