// Host harness for the quick phases of lg_crfloat.cuh with contracted
// products: the device's packed multiplies (crf_mulx) may be fused into a
// following packed add, so here a lane type remembers that it is such a
// product, and each add or subtraction of one that a bit of the mask names
// (in the order they are met) is a single fma.  Every function has to return
// the double evaluation rounded once whichever of them are fused.
//   crf_contract <points> <seed>
// prints: for each of exp log atan atanh pow polar, the sums met and the
// mismatches over all masks
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#define LG_CRF_HOST 1
#include "../../lensed_gb300/device/lg_crfloat.cuh"

struct lane {
    float v;
    float a, b;
    bool prod;
};
static unsigned g_mask = 0;
static int g_site = 0, g_sites = 0;
static bool fuse()
{
    const bool f = g_mask >> (g_site & 31) & 1;
    if (++g_site > g_sites) g_sites = g_site;
    return f;
}
static lane plain(float v) { return {v, 0.0f, 0.0f, false}; }
template <> struct crf_lanes<lane> { static const int n = 1; };
static inline void crf_fill(lane& v, float s) { v = plain(s); }
static inline float crf_get(const lane& v, int) { return v.v; }
static inline void crf_set(lane& v, int, float s) { v = plain(s); }
static inline lane crf_neg(lane a) { return {-a.v, -a.a, a.b, a.prod}; }
static inline lane crf_abs(lane a) { return plain(std::fabs(a.v)); }
static inline lane crf_mul(lane a, lane b) { return plain(a.v * b.v); }
static inline lane crf_mulx(lane a, lane b) { return {a.v * b.v, a.v, b.v, true}; }
static inline lane crf_fma(lane a, lane b, lane c) { return plain(std::fma(a.v, b.v, c.v)); }
static inline lane crf_add(lane a, lane b)
{
    if (a.prod && fuse()) return plain(std::fma(a.a, a.b, b.v));
    if (b.prod && fuse()) return plain(std::fma(b.a, b.b, a.v));
    return plain(a.v + b.v);
}
static inline lane crf_sub(lane a, lane b) { return crf_add(a, crf_neg(b)); }

static std::mt19937_64 g_rng;
static double uni(double lo, double hi) { return std::uniform_real_distribution<double>(lo, hi)(g_rng); }
static bool differ(float v, float w) { return v != w && !(v != v && w != w); }

// all masks of the sums that `one` meets
template <class Fn>
static void sweep(long n, Fn one)
{
    long bad = 0;
    g_sites = 0;
    g_mask = 0;
    for (long i = 0; i < 1000; ++i) g_site = 0, one(i);
    const int sites = g_sites;
    for (g_mask = 0; g_mask < 1u << sites; ++g_mask)
        for (long i = 0; i < n; ++i) {
            g_site = 0;
            bad += one(i);
        }
    std::printf("%d %ld\n", sites, bad);
}

int main(int argc, char** argv)
{
    if (argc != 3) return 2;
    const long n = std::atol(argv[1]);
    g_rng.seed(std::atol(argv[2]));
    sweep(n, [](long) {
        const float x = (float)uni(-87, 87);
        return differ(lg_crf_exp<lane>(plain(x)).v, (float)std::exp((double)x));
    });
    sweep(n, [](long i) {
        const float x = (float)std::exp2(uni(-90, 91) * (i % 2 ? 1 : 0.02));
        return differ(lg_crf_log<lane>(plain(x)).v, (float)std::log((double)x));
    });
    sweep(n, [](long i) {
        const float x = (float)(i % 4 ? uni(-2, 2) : std::exp2(uni(-12, 24)));
        return differ(lg_crf_atan<lane>(plain(x)).v, (float)std::atan((double)x));
    });
    sweep(n, [](long i) {
        const float x = (float)(i % 4 ? uni(-0.9, 0.9) : uni(-0.02, 0.02));
        return differ(lg_crf_atanh<lane>(plain(x)).v, (float)std::atanh((double)x));
    });
    static const float Y[] = {0.2f, -0.2f, 0.05f, -0.13f, 0.5f, 1.0f, -1.0f, 0.9f, 2.0f, -3.3f, 7.7f};
    sweep(n, [](long i) {
        const float x = (float)std::exp2(uni(-10, 10)), y = Y[i % 11];
        return differ(lg_crf_pow1<lane>(plain(x), y).v, (float)std::pow((double)x, (double)y));
    });
    sweep(n, [](long) {
        const float x = (float)uni(-200, 200), y = (float)uni(-200, 200);
        lane r, c, s, c2, s2;
        bool ok[2];
        crf_quick_polar<lane>(plain(x), plain(y), r, c, s, c2, s2, ok);
        if (!ok[0]) return false;
        const float phi = (float)std::atan2((double)y, (double)x), xx = x * x, yy = y * y;
        return r.v != std::sqrt(xx + yy) || c.v != (float)std::cos((double)phi) || s.v != (float)std::sin((double)phi) ||
               c2.v != (float)std::cos((double)(2 * phi)) || s2.v != (float)std::sin((double)(2 * phi));
    });
    return 0;
}
