// Diagnostic entry points: the paired-ray elementary functions of the
// device prelude (exp, log, square root, reciprocal, arctangent and inverse
// hyperbolic tangent used by the fast evaluation modules) and the correctly
// rounded functions of the exact modules (lg_crfloat.cuh), evaluated on a
// vector of inputs, so their accuracy can be checked against
// double-precision references on the host; and a sweep that compares the
// correctly rounded functions with the double evaluation on the device over
// a range of float bit patterns, or over points and powers made from them.

#include <cuda_runtime.h>

#include "lg_internal.h"
#include "../device/lg_prelude.cuh"
#define LG_CRF_SMEM 1
#include "../device/lg_crfloat.cuh"

namespace {

// correctly rounded function fn (0 exp, 1 log, 2 atan, 3 atanh) of a pair
__device__ float2 crf_pair(int fn, float2 a)
{
    return fn == 0 ? lg_crf_exp(a) : fn == 1 ? lg_crf_log(a) : fn == 2 ? lg_crf_atan(a) : lg_crf_atanh(a);
}
__device__ float crf_scalar(int fn, float x)
{
    return fn == 0 ? lg_crf_exp(x) : fn == 1 ? lg_crf_log(x) : fn == 2 ? lg_crf_atan(x) : lg_crf_atanh(x);
}
__device__ float crf_double(int fn, float x)
{
    return fn == 0   ? (float)exp((double)x)
           : fn == 1 ? (float)log((double)x)
           : fn == 2 ? (float)atan((double)x)
                     : (float)atanh((double)x);
}

// the EPL lens's functions, one value: fn 4 sin, 5 cos, 6 pow(x, Y[u % 16])
// with the lens's exponents and others, 7 atan2(x, p), 8 pow(|x|, p), p the
// float of bit pattern u * 0x9E3779B1 (the second argument swept too)
__constant__ float lg_probe_y[16] = {-1.2f, -1.0f, -0.8f, -0.5f, 0.5f, -0.25f, 0.2f, 1.0f / 3,
                                     2.5f, -2.2f, 0.999f, 1.5f, -0.1f, 3.7f, 0.05f, -7.5f};
__device__ float crf_two(int fn, float x, unsigned u)
{
    const float p = __uint_as_float(u * 0x9E3779B1u);
    float s, c;
    switch (fn) {
    case 4: lg_crf_sincos(x, &s, &c); return s;
    case 5: lg_crf_sincos(x, &s, &c); return c;
    case 6: return lg_crf_pow(x, lg_probe_y[u % 16]);
    case 7: return lg_crf_atan2(x, p);
    default: return lg_crf_pow(fabsf(x), p);
    }
}
__device__ float crf_two_double(int fn, float x, unsigned u)
{
    const float p = __uint_as_float(u * 0x9E3779B1u);
    switch (fn) {
    case 4: return (float)sin((double)x);
    case 5: return (float)cos((double)x);
    case 6: return (float)pow((double)x, (double)lg_probe_y[u % 16]);
    case 7: return (float)atan2((double)x, (double)p);
    default: return (float)pow((double)fabsf(x), (double)p);
    }
}

// The EPL lens's quick phases on a pair made from u by a bit mixer: fn 9 the
// polar frame (mismatches among its decided lanes), 10 the power with one
// exponent.  Points of sizes 2^-33 to
// 2^33 (a quarter of ordinary size), one in eight each near the x axis, the y
// axis and a diagonal, others with min/max near 2^-20; bases over the whole
// range of the quick logarithm and near 1, the lens's exponents and any up to
// 2^8.
__device__ unsigned long long probe_mix(unsigned long long z)
{
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
// a float of random sign and mantissa bits, of binary exponent e
__device__ float probe_float(unsigned h, int e) { return __uint_as_float((h & 0x807fffffu) | (unsigned)(e + 127) << 23); }
__device__ int quick_pair(int fn, unsigned u)
{
    float x[2], y[2];
    unsigned h = 0;
    for (int i = 0; i < 2; ++i) {
        const unsigned long long z = probe_mix(2ull * u + i + 0x9E3779B97F4A7C15ull);
        const unsigned a = (unsigned)z, b = (unsigned)(z >> 32);
        h = (unsigned)probe_mix(z);
        if (fn == 10) {
            x[i] = fabsf(probe_float(a, h % 2 ? (int)(b % 181) - 90 : (int)(b % 3) - 1));
            continue;
        }
        const int e = h % 4 == 0 ? 5 : (int)(h >> 8 & 63) - 31;
        x[i] = probe_float(a, e - (h >> 14 & 1));
        y[i] = probe_float(b, e - (h >> 15 & 1));
        const int kind = h >> 16 & 7, small = h >> 20 & 31;
        if (kind == 0) y[i] = probe_float(b, e - small < -120 ? -120 : e - small);
        if (kind == 1) x[i] = probe_float(a, e - small < -120 ? -120 : e - small);
        if (kind == 2) y[i] = (b & 1 ? x[i] : -x[i]) * (1.0f + (b >> 28) * 0x1p-23f);
        if (kind == 3) y[i] = x[i] * 0x1p-20f * (1.0f + ((int)(b >> 28) - 8) * 0x1p-23f);
    }
    const float2 X = make_float2(x[0], x[1]);
    auto same = [](float v, float w) { return __float_as_uint(v) == __float_as_uint(w) || (v != v && w != w); };
    if (fn == 10) {
        const float e = h & 1 ? lg_probe_y[h >> 1 & 15] : probe_float(h, (int)(h >> 23 & 15) - 7);
        const float2 r = lg_crf_pow1(X, e);
        return !same(r.x, (float)pow((double)x[0], (double)e)) + !same(r.y, (float)pow((double)x[1], (double)e));
    }
    float2 r, c, s, c2, s2;
    bool ok[2];
    crf_quick_polar(X, make_float2(y[0], y[1]), r, c, s, c2, s2, ok);
    int bad = 0;
    for (int i = 0; i < 2; ++i) {
        if (!ok[i]) continue;
        const float phi = (float)atan2((double)y[i], (double)x[i]);
        const float root = __fsqrt_rn(__fadd_rn(__fmul_rn(x[i], x[i]), __fmul_rn(y[i], y[i])));
        bad += !(same(crf_get(r, i), root) && same(crf_get(c, i), (float)cos((double)phi)) &&
                 same(crf_get(s, i), (float)sin((double)phi)) && same(crf_get(c2, i), (float)cos((double)(2 * phi))) &&
                 same(crf_get(s2, i), (float)sin((double)(2 * phi))));
    }
    return bad;
}

// every bit pattern u in [lo, hi) as lane 0 of a pair whose lane 1 is an
// unrelated input (u times an odd constant, a bijection of the 32-bit
// patterns), so that the lanes of a pair take different paths and table
// entries, and through the one-lane version; counts inputs whose bits
// differ from the double evaluation in either (NaN equal to NaN), and
// keeps the first few
__global__ void lg_crf_sweep_kernel(int fn, unsigned long long lo, unsigned long long hi,
                                    unsigned long long* __restrict__ bad, unsigned* __restrict__ first, int nfirst)
{
    crf_load_tables<256>(threadIdx.x);
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    unsigned long long nbad = 0;
    for (unsigned long long u = lo + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; u < hi; u += stride) {
        const float x0 = __uint_as_float((unsigned)u);
        if (fn >= 9) {
            const int n = quick_pair(fn, (unsigned)u);
            if (n) {
                nbad += n;
                const unsigned long long k = atomicAdd(bad + 1, 1ull);
                if (k < (unsigned long long)nfirst) first[k] = (unsigned)u;
            }
            continue;
        }
        if (fn >= 4) {
            const float r0 = crf_two(fn, x0, (unsigned)u), w0 = crf_two_double(fn, x0, (unsigned)u);
            if (!(__float_as_uint(r0) == __float_as_uint(w0) || (r0 != r0 && w0 != w0))) {
                ++nbad;
                const unsigned long long k = atomicAdd(bad + 1, 1ull);
                if (k < (unsigned long long)nfirst) first[k] = (unsigned)u;
            }
            continue;
        }
        const float x1 = __uint_as_float((unsigned)u * 0x9E3779B1u);
        const float2 r = crf_pair(fn, make_float2(x0, x1));
        const float w0 = crf_double(fn, x0), w1 = crf_double(fn, x1);
        // the one-lane version (what the exact render calls) on x0 too
        const float r0 = crf_scalar(fn, x0);
        const bool ok0 = (__float_as_uint(r.x) == __float_as_uint(w0) || (r.x != r.x && w0 != w0)) &&
                         (__float_as_uint(r0) == __float_as_uint(w0) || (r0 != r0 && w0 != w0));
        const bool ok1 = __float_as_uint(r.y) == __float_as_uint(w1) || (r.y != r.y && w1 != w1);
        if (!ok0 || !ok1) {
            nbad += (!ok0) + (!ok1);
            const unsigned long long k = atomicAdd(bad + 1, 1ull);
            if (k < (unsigned long long)nfirst) first[k] = ok0 ? __float_as_uint(x1) : (unsigned)u;
        }
    }
    if (nbad) atomicAdd(bad, nbad);
}

__global__ void lg_pair_math_kernel(int fn, const float* __restrict__ x, int n, float* __restrict__ out)
{
    crf_load_tables<256>(threadIdx.x);
    const int i = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= n) return;
    const lg_pair a = lg_pair_of(x[i], i + 1 < n ? x[i + 1] : 1.0f);
    const lg_pair r = fn == 0   ? expf(a)
                      : fn == 1 ? logf(a)
                      : fn == 2 ? sqrtf(a)
                      : fn == 3 ? 1.0f / a
                      : fn == 4 ? atanf(a)
                      : fn == 5 ? atanhf(a)
                                : lg_pair{crf_pair(fn - 6, a.v)};
    out[i] = r.v.x;
    if (i + 1 < n) out[i + 1] = r.v.y;
}

}  // namespace

extern "C" int lg_probe_pair_math(int device, int fn, const float* x, int n, float* out)
{
    if (!x || !out || n < 0 || fn < 0 || fn > 9) return LG_ERR_INPUT;
    if (n == 0) return LG_OK;
    auto fail = [](cudaError_t e) {
        lg::set_global_error(cudaGetErrorString(e));
        return LG_ERR_CUDA;
    };
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return fail(e);
    float *dx = nullptr, *dy = nullptr;
    const size_t bytes = (size_t)n * 4;
    if ((e = cudaMalloc((void**)&dx, bytes)) != cudaSuccess) return fail(e);
    if ((e = cudaMalloc((void**)&dy, bytes)) != cudaSuccess) {
        cudaFree(dx);
        return fail(e);
    }
    e = cudaMemcpy(dx, x, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        const int pairs = (n + 1) / 2;
        lg_pair_math_kernel<<<(pairs + 255) / 256, 256>>>(fn, dx, n, dy);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, dy, bytes, cudaMemcpyDeviceToHost);
    cudaFree(dx);
    cudaFree(dy);
    return e == cudaSuccess ? LG_OK : fail(e);
}

extern "C" int lg_probe_crf_sweep(int device, int fn, unsigned long long lo, unsigned long long hi,
                                  unsigned long long* mismatches, unsigned* first, int nfirst)
{
    if (fn < 0 || fn > 10 || lo > hi || hi > (1ull << 32) || !mismatches || nfirst < 0 || (nfirst && !first))
        return LG_ERR_INPUT;
    auto fail = [](cudaError_t e) {
        lg::set_global_error(cudaGetErrorString(e));
        return LG_ERR_CUDA;
    };
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return fail(e);
    unsigned long long* d_bad = nullptr;
    unsigned* d_first = nullptr;
    if ((e = cudaMalloc((void**)&d_bad, 2 * sizeof(unsigned long long))) != cudaSuccess) return fail(e);
    if ((e = cudaMalloc((void**)&d_first, (nfirst ? nfirst : 1) * sizeof(unsigned))) != cudaSuccess) {
        cudaFree(d_bad);
        return fail(e);
    }
    e = cudaMemset(d_bad, 0, 2 * sizeof(unsigned long long));
    if (e == cudaSuccess && hi > lo) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        lg_crf_sweep_kernel<<<sms * 8, 256>>>(fn, lo, hi, d_bad, d_first, nfirst);
        e = cudaGetLastError();
    }
    unsigned long long h[2] = {0, 0};
    if (e == cudaSuccess) e = cudaMemcpy(h, d_bad, sizeof h, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && nfirst)
        e = cudaMemcpy(first, d_first, (size_t)(h[1] < (unsigned long long)nfirst ? h[1] : nfirst) * sizeof(unsigned),
                       cudaMemcpyDeviceToHost);
    cudaFree(d_bad);
    cudaFree(d_first);
    if (e != cudaSuccess) return fail(e);
    *mismatches = h[0];
    return LG_OK;
}
