// Host check of sl_parts.cuh: differences of FP64 positions in three FP32
// parts against the exact difference, in units of the FP32 last place of the
// exact difference.  Positions at several distances from the origin, pairs a
// few radii apart, components much smaller than that, equal ones, opposite
// signs and neighbours of powers of two.  Prints "<distance> <cases> <max error>".
#include "sl_parts.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

static std::mt19937_64 rng(99);
static double uniform(double lo, double hi) { return std::uniform_real_distribution<double>(lo, hi)(rng); }

struct Parts {
    float p[3];
};

static Parts split(double x)  // the drift kernel's
{
    const float hi = (float)x;
    const double rem = x - hi;
    const float lo = sl::parts::grid_part(hi, (float)rem);
    return {{hi, lo, (float)(rem - lo)}};
}

int main(int argc, char** argv)
{
    const long n = argc > 1 ? atol(argv[1]) : 1000000;
    const double distance[] = {0, 50, 1e4, 1e6, 1e8};
    for (double X : distance) {
        double worst = 0;
        for (long i = 0; i < n; ++i) {
            const double scale = X == 0 ? 50 : X;
            double a = uniform(-scale, scale), b;
            if (i % 7 == 0) a = std::ldexp(rng() & 1 ? 1.0 : -1.0, (int)std::floor(std::log2(scale))) * (1 + uniform(-1e-7, 1e-7));
            switch (i % 5) {
            case 0: b = a + uniform(-3, 3); break;
            case 1: b = a + uniform(-3, 3) * std::ldexp(1.0, -(int)(rng() % 20)); break;
            case 2: b = -a + uniform(-3, 3); break;
            case 3: b = uniform(-scale, scale); break;
            default: b = rng() & 1 ? a : std::nextafter(a, 2 * a); break;
            }
            const Parts pa = split(a), pb = split(b);
            const float r = sl::parts::sub3(pa.p[0], pa.p[1], pa.p[2], pb.p[0], pb.p[1], pb.p[2]);
            // a - b = d + rest exactly (TwoSum)
            const double d = a - b, bp = d - a, rest = (a - (d - bp)) - (b + bp);
            if (d == 0) {
                if (r != 0) worst = INFINITY;
                continue;
            }
            int e;
            std::frexp(d, &e);
            const double err = std::fabs((r - d) - rest) / std::ldexp(1.0, e - 24);
            worst = err > worst ? err : worst;
        }
        std::printf("%g %ld %.6f\n", X, n, worst);
    }
    return 0;
}
