// Host harness for lg_crf_pow1 where its error is largest: bases whose quick
// logarithm's float part is furthest off, exponents whose result lies just below a power
// of two (there the error counts most against the rounding), and the
// arguments given on the command line.
//   crf_pow <bases> <seed> [<x> <y>]...
// prints: powers mismatches
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#define LG_CRF_HOST 1
#include "../../lensed_gb300/device/lg_crfloat.cuh"

static long g_n = 0, g_bad = 0;
static void check(float x, float y)
{
    ++g_n;
    if (lg_crf_pow1<float>(x, y) != (float)std::pow((double)x, (double)y) && g_bad++ < 8)
        std::fprintf(stderr, "%a ^ %a\n", x, y);
}

int main(int argc, char** argv)
{
    if (argc < 3) return 2;
    for (int i = 3; i + 1 < argc; i += 2) check(std::strtof(argv[i], nullptr), std::strtof(argv[i + 1], nullptr));
    std::mt19937_64 g(std::atol(argv[2]));
    std::uniform_real_distribution<double> u(0, 1);
    for (long i = 0, n = std::atol(argv[1]); i < n; ++i) {
        const float x = (float)std::exp((u(g) * 2 - 1) * (i % 3 == 0 ? 62 : i % 3 == 1 ? 2 : 0.5));
        float s1, r, t, e;
        crf_quick_log<float>(x, s1, r, t, e);
        const double ln = std::log((double)x), a = r + (t - 0x1.6p-34f);
        if (std::fabs((double)s1 - ln + a) < 0x1.4p-34) continue;
        const double top = std::fmin(300.0, 85 / std::fabs(ln));
        for (int k = 0; k < 4000; ++k) {
            const double m = std::floor((u(g) * 2 - 1) * top * std::fabs(ln) / M_LN2);
            check(x, (float)((m - 0.05 * u(g)) * M_LN2 / ln));
        }
    }
    std::printf("%ld %ld\n", g_n, g_bad);
    return 0;
}
