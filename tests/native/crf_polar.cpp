// Host harness for the EPL lens's quick phases (lg_crfloat.cuh with
// LG_CRF_HOST): random points through crf_quick_polar (r, cos, sin of phi =
// atan2 rounded, of 2 phi) and random bases through lg_crf_pow1, each
// compared with the functions evaluated in double and rounded once.
//   crf_polar <points> <log2 of the size range> <seed>
// prints: points polar_mismatches polar_undecided pow_mismatches pow_rest
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

static long g_rest = 0;
#define LG_CRF_REST_COUNT() (++g_rest)
#define LG_CRF_HOST 1
#include "../../lensed_gb300/device/lg_crfloat.cuh"

int main(int argc, char** argv)
{
    if (argc != 4) return 2;
    const long n = std::atol(argv[1]);
    const double range = std::atof(argv[2]);
    std::mt19937_64 g(std::atol(argv[3]));
    std::uniform_real_distribution<double> u(-1, 1);
    static const float Y[] = {0.2f, -0.2f, 0.05f, -0.13f, 0.5f, 1.0f, -1.0f, 0.9f, 2.0f, -3.3f, 0.0f, 7.7f};
    long bad = 0, und = 0, pbad = 0, prest = 0;
    for (long i = 0; i < n; ++i) {
        const double size = std::exp2(u(g) * range);
        float x = (float)(u(g) * size), y = (float)(u(g) * size);
        // near an axis, on one, on a diagonal
        if (i % 8 == 1) y *= (float)std::exp2(-24 * std::fabs(u(g)));
        if (i % 8 == 2) x *= (float)std::exp2(-24 * std::fabs(u(g)));
        if (i % 512 == 3) y = 0.0f;
        if (i % 512 == 4) x = -0.0f;
        if (i % 64 == 5) y = i % 128 == 5 ? x : -x;
        float r, c, s, c2, s2;
        bool ok[2];
        crf_quick_polar<float>(x, y, r, c, s, c2, s2, ok);
        und += !ok[0];
        if (ok[0]) {
            const float phi = (float)std::atan2((double)y, (double)x);
            const float xx = x * x, yy = y * y;
            bad += r != std::sqrt(xx + yy) || c != (float)std::cos((double)phi) || s != (float)std::sin((double)phi) ||
                   c2 != (float)std::cos((double)(2 * phi)) || s2 != (float)std::sin((double)(2 * phi));
        }
        const float e = Y[i % 12], b = (float)std::exp2(u(g) * range);
        const long r0 = g_rest;
        const float v = lg_crf_pow1<float>(b, e), w = (float)std::pow((double)b, (double)e);
        pbad += v != w && !(v != v && w != w);
        prest += g_rest - r0;
    }
    std::printf("%ld %ld %ld %ld %ld\n", n, bad, und, pbad, prest);
    return 0;
}
