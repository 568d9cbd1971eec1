// Correctly rounded single-precision exp, log, atan, atanh, sin, cos, pow
// and atan2 computed in single-precision arithmetic, for the exact
// evaluation modules.
//
// The likelihood's FP32 semantics (the oracle's, and the strict modules')
// takes every elementary function as its value evaluated in double and
// rounded once to float.  GB300 executes FP64 at a small fraction of its
// FP32 rate, so per ray these functions are computed here instead with
// "double-word" arithmetic -- a value carried as an unevaluated sum hi + lo
// of two floats, with exact products and sums from fma (Dekker 1971, "A
// floating-point technique for extending the available precision") -- after
// table-driven argument reductions (Tang 1989, "Table-driven implementation
// of the exponential function in IEEE floating-point arithmetic"; Tang 1990,
// "... of the logarithm function").  The double-word result is within about
// 2^-42 of the true value (relative); Ziv's rounding test (Ziv 1991, "Fast
// evaluation of elementary mathematical functions with correctly rounded
// last bit") then rounds both ends of that error interval, and if they round
// to the same float, that float is the correctly rounded result -- which is
// also what the double evaluation rounds to, its own error being far smaller
// than the interval.  Otherwise (about one call in 2^16) the lane evaluates
// the function in double and rounds once, exactly as the strict modules do.
// So each function returns the double-then-round value for every input (the
// bounds are in the comments; all 2^32 inputs of the one-argument functions
// have been compared, the others on samples).
//
// exp, log, atan and atanh first take a quick phase (below), whose error is
// a few 2^-35 to 2^-39 and whose own rounding test leaves one lane in 2^9 to
// 2^13 to the full phase.  The quick phases are written once over a lane
// type F: float (one value; also compiled for the host, with LG_CRF_HOST,
// for the CPU tests) or float2 (two rays, with the paired f32x2
// instructions); the full phases take one value at a time.  Every operation
// is a single IEEE round-to-nearest operation (no contraction is left to the
// compiler).  Tables: lg_crf_tables.cuh and lg_crf_consts.cuh, generated by
// make_crf_tables.py.

#ifdef LG_CRF_HOST
#include <cmath>
#include <cstdint>
#include <cstring>
#define LG_CRF_DEV static inline
#define LG_CRF_COLD static
#define LG_CRF_TABLE(name, n) static const unsigned long long name[n]
struct float2 {
    float x, y;
};
struct float4 {
    float x, y, z, w;
};
#else
#define LG_CRF_DEV static __device__ __forceinline__
#define LG_CRF_COLD static __device__ __noinline__
#define LG_CRF_TABLE(name, n) __device__ const __align__(16) unsigned long long name[n]
#endif

// ------------------------------------------------------------- primitives --
#ifdef LG_CRF_HOST
LG_CRF_DEV float crf_add(float a, float b) { return a + b; }
LG_CRF_DEV float crf_sub(float a, float b) { return a - b; }
LG_CRF_DEV float crf_mul(float a, float b) { return a * b; }
LG_CRF_DEV float crf_fma(float a, float b, float c) { return std::fma(a, b, c); }
LG_CRF_DEV int crf_bits(float a)
{
    int i;
    std::memcpy(&i, &a, 4);
    return i;
}
LG_CRF_DEV float crf_from_bits(int i)
{
    float a;
    std::memcpy(&a, &i, 4);
    return a;
}
// reciprocal estimate: any value within a few ulp of 1/a serves (the
// double-word steps correct it); the host uses the IEEE quotient unless a
// test build substitutes a perturbed one (to stand in for the device's
// approximate reciprocal)
#ifndef LG_CRF_HOST_RCP
#define LG_CRF_HOST_RCP(a) (1.0f / (a))
#endif
LG_CRF_DEV float crf_rcp(float a) { return LG_CRF_HOST_RCP(a); }
LG_CRF_DEV float crf_rsqrt(float a) { return LG_CRF_HOST_RCP(std::sqrt(a)); }
// (a test build may count the lanes that take the double path)
#ifndef LG_CRF_SLOW_COUNT
#define LG_CRF_SLOW_COUNT()
#endif
// integer fields of the arguments' bit patterns (see the device versions)
LG_CRF_DEV void crf_log_fields(int b, int& e, int& j, int& mb)
{
    const int t = b - 0x3f400000;
    e = t >> 23;
    j = (t >> 13) & 1023;
    mb = b - e * 0x800000;
}
LG_CRF_DEV void crf_exp_fields(int bits, int& j, int& m)
{
    const int k = bits - 0x4b400000;
    j = k & 63;
    m = k >> 6;
}
LG_CRF_DEV int crf_pow2_bits(int e) { return (e + 127) * 0x800000; }   // bits of 2^e (normal e)
LG_CRF_DEV int crf_add_exp(int bits, int m) { return bits + m * 0x800000; }
LG_CRF_DEV float crf_slow_exp(float x) { LG_CRF_SLOW_COUNT(); return (float)std::exp((double)x); }
LG_CRF_DEV float crf_slow_log(float x) { LG_CRF_SLOW_COUNT(); return (float)std::log((double)x); }
LG_CRF_DEV float crf_slow_atan(float x) { LG_CRF_SLOW_COUNT(); return (float)std::atan((double)x); }
LG_CRF_DEV float crf_slow_atanh(float x) { LG_CRF_SLOW_COUNT(); return (float)std::atanh((double)x); }
LG_CRF_DEV float crf_slow_sin(float x) { LG_CRF_SLOW_COUNT(); return (float)std::sin((double)x); }
LG_CRF_DEV float crf_slow_cos(float x) { LG_CRF_SLOW_COUNT(); return (float)std::cos((double)x); }
LG_CRF_DEV float crf_slow_pow(float x, float y) { LG_CRF_SLOW_COUNT(); return (float)std::pow((double)x, (double)y); }
LG_CRF_DEV float crf_slow_atan2(float y, float x)
{
    LG_CRF_SLOW_COUNT();
    return (float)std::atan2((double)y, (double)x);
}
#else
LG_CRF_DEV float crf_add(float a, float b) { return __fadd_rn(a, b); }
LG_CRF_DEV float crf_sub(float a, float b) { return __fsub_rn(a, b); }
LG_CRF_DEV float crf_mul(float a, float b) { return __fmul_rn(a, b); }
LG_CRF_DEV float crf_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
// paired operations on f32x2.  With CUDA 13.0 the assembler fused an f32x2
// multiply into a following f32x2 add (also without contraction), so a
// product that must be rounded first is an fma with -0 (the same value for
// every operand), read from memory so that the assembler cannot see it.
// Negated and absolute operands are free (instruction modifiers).
__constant__ float2 crf_negzero = {-0.0f, -0.0f};
LG_CRF_DEV float2 crf_mul(float2 a, float2 b) { return __ffma2_rn(a, b, crf_negzero); }
LG_CRF_DEV float2 crf_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
LG_CRF_DEV float2 crf_sub(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
LG_CRF_DEV float2 crf_fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
LG_CRF_DEV int crf_bits(float a) { return __float_as_int(a); }
LG_CRF_DEV float crf_from_bits(int i) { return __int_as_float(i); }
// PTX rcp.approx (within about 1 ulp; subnormal results flushed, which
// the callers tolerate: see each use)
LG_CRF_DEV float crf_rcp(float a)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}
// PTX rsqrt.approx (within about 2 ulp)
LG_CRF_DEV float crf_rsqrt(float a)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}
// Integer fields of the arguments' bit patterns, in inline PTX: with CUDA
// 13.0 the optimizer was seen to miscompute such per-lane shifts of paired
// values (a lane's t >> 23 came out as t), and an asm block is opaque to it.
//   log: t = b - bits(0.75); e = t >> 23 (arithmetic); j = (t >> 13) & 1023;
//        mb = b - e 2^23 (the mantissa scaled into [0.75, 1.5))
LG_CRF_DEV void crf_log_fields(int b, int& e, int& j, int& mb)
{
    asm("{\n.reg .s32 t, x;\nsub.s32 t, %3, 0x3f400000;\nshr.s32 %0, t, 23;\nshr.s32 x, t, 13;\n"
        "and.b32 %1, x, 1023;\nshl.b32 x, %0, 23;\nsub.s32 %2, %3, x;\n}"
        : "=r"(e), "=r"(j), "=r"(mb)
        : "r"(b));
}
//   exp: k = bits - bits(1.5 2^23); j = k & 63; m = k >> 6 (arithmetic)
LG_CRF_DEV void crf_exp_fields(int bits, int& j, int& m)
{
    asm("{\n.reg .s32 k;\nsub.s32 k, %2, 0x4b400000;\nand.b32 %0, k, 63;\nshr.s32 %1, k, 6;\n}"
        : "=r"(j), "=r"(m)
        : "r"(bits));
}
// bits of 2^e for a normal power of two, and bits + m 2^23 (a float scaled
// by 2^m while it stays normal)
LG_CRF_DEV int crf_pow2_bits(int e)
{
    int r;
    asm("{\n.reg .s32 x;\nadd.s32 x, %1, 127;\nshl.b32 %0, x, 23;\n}" : "=r"(r) : "r"(e));
    return r;
}
LG_CRF_DEV int crf_add_exp(int bits, int m)
{
    int r;
    asm("{\n.reg .s32 x;\nshl.b32 x, %2, 23;\nadd.s32 %0, %1, x;\n}" : "=r"(r) : "r"(bits), "r"(m));
    return r;
}
// the lanes the double-word path cannot decide: the function in double,
// rounded once (out of line: a cold path)
LG_CRF_COLD float crf_slow_exp(float x) { return (float)exp((double)x); }
LG_CRF_COLD float crf_slow_log(float x) { return (float)log((double)x); }
LG_CRF_COLD float crf_slow_atan(float x) { return (float)atan((double)x); }
LG_CRF_COLD float crf_slow_atanh(float x) { return (float)atanh((double)x); }
LG_CRF_COLD float crf_slow_sin(float x) { return (float)sin((double)x); }
LG_CRF_COLD float crf_slow_cos(float x) { return (float)cos((double)x); }
LG_CRF_COLD float crf_slow_pow(float x, float y) { return (float)pow((double)x, (double)y); }
LG_CRF_COLD float crf_slow_atan2(float y, float x) { return (float)atan2((double)y, (double)x); }
LG_CRF_DEV float crf_get(float2 v, int i) { return i ? v.y : v.x; }
LG_CRF_DEV void crf_set(float2& v, int i, float s)
{
    if (i)
        v.y = s;
    else
        v.x = s;
}
// entry j of a table of float pairs (quads)
LG_CRF_DEV float2 crf_tab2(const unsigned long long* t, int j) { return __ldg(reinterpret_cast<const float2*>(t) + j); }
LG_CRF_DEV float4 crf_tab4(const unsigned long long* t, int j) { return __ldg(reinterpret_cast<const float4*>(t) + j); }
#endif

#ifdef LG_CRF_HOST
LG_CRF_DEV float2 crf_tab2(const unsigned long long* t, int j)
{
    float2 v;
    std::memcpy(&v, t + j, 8);
    return v;
}
LG_CRF_DEV float4 crf_tab4(const unsigned long long* t, int j)
{
    float4 v;
    std::memcpy(&v, t + 2 * j, 16);
    return v;
}
LG_CRF_DEV float crf_fabsf(float a) { return std::fabs(a); }
LG_CRF_DEV float crf_copysignf(float a, float b) { return std::copysign(a, b); }
#else
LG_CRF_DEV float crf_fabsf(float a) { return fabsf(a); }
LG_CRF_DEV float crf_copysignf(float a, float b) { return copysignf(a, b); }
#endif
LG_CRF_DEV float crf_get(float v, int) { return v; }
LG_CRF_DEV void crf_set(float& v, int, float s) { v = s; }

template <class F> struct crf_lanes;
template <> struct crf_lanes<float> { static const int n = 1; };
template <> struct crf_lanes<float2> { static const int n = 2; };

LG_CRF_DEV void crf_fill(float& v, float s) { v = s; }
LG_CRF_DEV void crf_fill(float2& v, float s)
{
    v.x = s;
    v.y = s;
}
// s in every lane
template <class F>
LG_CRF_DEV F crf_bc(float s)
{
    F v;
    crf_fill(v, s);
    return v;
}
LG_CRF_DEV float crf_neg(float a) { return -a; }
LG_CRF_DEV float2 crf_neg(float2 a)
{
    float2 v;
    v.x = -a.x;
    v.y = -a.y;
    return v;
}
LG_CRF_DEV float crf_abs(float a) { return crf_fabsf(a); }
LG_CRF_DEV float2 crf_abs(float2 a)
{
    float2 v;
    v.x = crf_fabsf(a.x);
    v.y = crf_fabsf(a.y);
    return v;
}

// (the library embeds the constants here for NVRTC, which has no include path)
#ifndef LG_CRF_CONSTS_INLINE
#include "lg_crf_consts.cuh"
#endif
// The tables: the array itself, or in NVRTC modules (LG_CRF_MODULE) a pointer
// to the library's copy on the device, which the host stores after loading
// the module.
#ifdef LG_CRF_MODULE
extern "C" __device__ const unsigned long long* lg_crf_base;
__device__ const unsigned long long* lg_crf_base;
#define LG_CRF_WORDS lg_crf_base
#else
#include "lg_crf_tables.cuh"
#define LG_CRF_WORDS lg_crf_words
#endif
#define lg_crf_exp_tab (LG_CRF_WORDS + LG_CRF_AT_EXP)
#define lg_crf_log_tab (LG_CRF_WORDS + LG_CRF_AT_LOG)
#define lg_crf_sc_tab (LG_CRF_WORDS + LG_CRF_AT_SC)
#define lg_crf_q_tab (LG_CRF_WORDS + LG_CRF_AT_Q)

// Entry of a quick-phase table: base (LG_CRF_Q_*) plus a byte offset.  With
// LG_CRF_SMEM the tables (28.7 KB) are read from a copy in shared memory that
// the kernel fills with crf_load_tables first: a lookup is then two or three
// instructions (32-bit offsets, the table's address an immediate) instead of
// the five of a global load with its 64-bit address, and the table reads are
// a fifth of the quick phases' instructions.
#if defined(LG_CRF_HOST)
LG_CRF_DEV float2 crf_qtab(int base, unsigned off)
{
    float2 v;
    std::memcpy(&v, lg_crf_q_tab + base + off / 8, 8);
    return v;
}
#elif defined(LG_CRF_SMEM)
__shared__ __align__(16) unsigned long long lg_crf_s[LG_CRF_Q_ENTRIES];
LG_CRF_DEV float2 crf_qtab(int base, unsigned off)
{
    return *reinterpret_cast<const float2*>(reinterpret_cast<const char*>(lg_crf_s) + 8 * base + off);
}
// every thread of the block (NT threads) calls it, before any lookup
template <int NT>
LG_CRF_DEV void crf_load_tables(int tid)
{
    const float4* src = reinterpret_cast<const float4*>(lg_crf_q_tab);
    float4* dst = reinterpret_cast<float4*>(lg_crf_s);
#pragma unroll 4
    for (int i = tid; i < LG_CRF_Q_ENTRIES / 2; i += NT) dst[i] = __ldg(src + i);
    __syncthreads();
}
#else
LG_CRF_DEV float2 crf_qtab(int base, unsigned off)
{
    return __ldg(reinterpret_cast<const float2*>(reinterpret_cast<const char*>(lg_crf_q_tab) + 8 * base + off));
}
#endif

// Relative half-width of Ziv's interval: the double-word results of the
// functions below are within 2^-42 of the true value (bound from the
// error analysis in each function; tests/test_crfloat.py measures it over
// all or dense samples of the inputs), so a margin of 2^-40 leaves a factor
// of 4.
#ifndef LG_CRF_ZIV
#define LG_CRF_ZIV (0x1p-40f)
#endif

// Both ends of [hi + lo - d, hi + lo + d], d = |hi| 2^-40, rounded: equal
// means the result.  (lo +- hi 2^-40 from an fma: the product is exact, a
// power-of-two scaling; for negative hi the two ends swap, which the
// equality test does not mind.)
LG_CRF_DEV void crf_ziv(float hi, float lo, float& z1, float& z2)
{
    z1 = crf_add(hi, crf_fma(hi, LG_CRF_ZIV, lo));
    z2 = crf_add(hi, crf_fma(hi, -LG_CRF_ZIV, lo));
}

// every lane of v satisfies ok
template <class F>
LG_CRF_DEV bool crf_all(const bool (&ok)[2])
{
    bool a = true;
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) a = a && ok[i];
    return a;
}

// ---------------------------------------------------------------------- exp --
// x = k ln2/64 + r, |r| <= ln2/128 (k = m 64 + j); e^x = 2^m 2^(j/64) e^r.
// r = x - k L_hi exactly (an fma: the difference is a multiple of 2^-31
// below 2^-7 in magnitude) minus k L_lo; e^r = 1 + r + r^2/2 + r^3 (1/6 +
// r/24) with r = rh + rl, the square of rh exact (fma), rl to first order
// (it reaches 2^-22), the cubic tail in float.
// Error: k L_lo rounding and the L_hi + L_lo split (2^-46 at |k| <= 9600),
// truncation r^5/120 (2^-44.6), table pairs (2^-48), evaluation (2^-47).
// Results below 2^-126 are rounded to the subnormal grid from the
// double-word value directly; e^x rounds to 0 for x <= LG_CRF_EXP_ZERO.
LG_CRF_COLD float crf_exp_low(float x, float yh0, float yl0, int m)
{
    // renormalise the pair (yl0 reaches a few ulp of yh0): |yl| <= ulp(yh)/2
    const float yh = crf_add(yh0, yl0);
    const float yl = crf_sub(yl0, crf_sub(yh, yh0));
    // the result y 2^m with m <= -126 and y < 2^(-126 - m): round y to the
    // grid g = 2^(-149 - m) with the magic number M = 2^(-126 - m), for
    // which M + y lies in [M, 2M) where floats are spaced by g
    const float M = crf_from_bits(crf_pow2_bits(-126 - m));
    const float g = crf_mul(M, 0x1p-23f), h = crf_mul(g, 0.5f);
    const float a = crf_add(M, yh);
    const float base = crf_sub(a, M);   // exact
    const float ea = crf_sub(yh, base);  // exact
    const float rho = crf_add(ea, yl);
    const float dd = crf_add(crf_mul(yh, LG_CRF_ZIV), crf_mul(h, 0x1p-22f));
    const float ar = crf_fabsf(rho);
    float q;
    if (ar < crf_sub(h, dd))
        q = base;
    else if (ar > crf_add(h, dd))
        q = crf_add(base, rho > 0.0f ? g : crf_neg(g));
    else
        return crf_slow_exp(x);
    // q 2^m, exactly, in two power-of-two steps (m + 64 >= -87)
    return crf_mul(crf_mul(q, crf_from_bits(crf_pow2_bits(m + 64))), 0x1p-64f);
}

// e^r 2^(j/64) as yh + yl for r = rh + rl (|rh| <= ln2/128 + 2^-17, rl to
// first order) and j, m (k = 64 m + j) from big = k + 1.5 2^23.
LG_CRF_DEV void crf_exp_tail(float big, float rh, float rl, float& yh, float& yl, int& m)
{
    const float sh = crf_mul(rh, rh);
    const float sl = crf_fma(rh, rh, crf_neg(sh));
    const float p3 = crf_fma(rh, 0x1.555556p-5f, 0x1.555556p-3f);
    const float h = crf_mul(sh, 0.5f);
    // first order in rl (up to 2^-22 at large |k|): rl (1 + rh + rh^2/2)
    const float small = crf_fma(crf_mul(sh, rh), p3, crf_fma(sl, 0.5f, crf_fma(h, rl, crf_fma(rh, rl, rl))));
    const float uh = crf_add(rh, h);  // |rh| >= rh^2 / 2: fast two-sum
    const float ul = crf_add(crf_sub(h, crf_sub(uh, rh)), small);
    int j;
    crf_exp_fields(crf_bits(big), j, m);
    const float2 T = crf_tab2(lg_crf_exp_tab, j);
    const float th = T.x, tl = T.y;
    // T (1 + u) = T + T uh + (T ul + tl uh + tl)
    const float ph = crf_mul(th, uh);
    const float pl = crf_fma(th, uh, crf_neg(ph));
    const float e = crf_add(crf_fma(th, ul, crf_fma(tl, uh, tl)), pl);
    yh = crf_add(th, ph);  // |th| >= 1 > |ph|: fast two-sum
    yl = crf_add(crf_sub(ph, crf_sub(yh, th)), e);
}

LG_CRF_DEV float crf_full_exp(float x)
{
    const float S = 0x1.8p23f;
    const float big = crf_fma(x, LG_CRF_EXP_INVL, S);  // k + 1.5 2^23 (|k| < 2^22)
    const float kf = crf_sub(big, S);
    const float rh = crf_fma(crf_neg(kf), LG_CRF_EXP_LHI, x);
    const float rl = crf_mul(crf_neg(kf), LG_CRF_EXP_LLO);
    float yh, yl, z1, z2;
    int m;
    crf_exp_tail(big, rh, rl, yh, yl, m);
    crf_ziv(yh, yl, z1, z2);
    if (x <= 88.0f && x > LG_CRF_EXP_ZERO) {
        if (m >= -125 || (m == -126 && z1 >= 1.0f))
            return z1 == z2 ? crf_from_bits(crf_add_exp(crf_bits(z1), m)) : crf_slow_exp(x);
        return crf_exp_low(x, yh, yl, m);
    }
    return x <= LG_CRF_EXP_ZERO ? 0.0f : crf_slow_exp(x);  // NaN, x > 88: in double
}

// ---------------------------------------------------------------------- log --
// log1p of the double-word r = rh + rl (|r| <= 2^-10): r - r^2/2 + r^3
// (1/3 - r/4 + r^2/5), the square exact; truncation r^6/6 (relative 2^-52
// where the result is r itself), the cubic term in float (relative to r,
// 3 roundings of a term below 2^-21.6: 2^-44).  Out: uh + ul.
LG_CRF_DEV void crf_log1p_dw(float rh, float rl, float& uh, float& ul)
{
    const float sh = crf_mul(rh, rh);
    const float sl = crf_fma(rh, rh, crf_neg(sh));
    const float P = crf_fma(crf_fma(rh, 0x1.99999ap-3f, -0.25f), rh, 0x1.555556p-2f);
    const float t = crf_mul(crf_mul(sh, rh), P);
    // r_lo - r_h r_lo - s_lo / 2 + t
    const float small = crf_add(crf_fma(crf_neg(rh), rl, rl), crf_fma(sl, -0.5f, t));
    const float h = crf_mul(sh, -0.5f);
    uh = crf_add(rh, h);  // |rh| >= rh^2 / 2: fast two-sum
    ul = crf_add(crf_sub(h, crf_sub(uh, rh)), small);
}

// ln(u), u = uh + ul > 0 (uh normal, |ul| <= ulp(uh)): u = 2^e m (m in
// [0.75, 1.5)) and m c_j = 1 + r with c_j from the table of the interval of
// m (|r| <= 2^-10), so ln u = e ln2 - ln(c_j) + log1p(r).  r = m c_j - 1 is exact as
// (m_hi c_j - 1) + (the product's rounding error) + m_lo c_j (the first term
// exactly by Sterbenz); c_j = 1 next to 1, so small logarithms keep their
// relative accuracy.  Sum: e ln2 as an exact product pair plus e LN2_LO,
// then two fast two-sums (|e ln2| >= |ln c_j| >= |log1p(r)| or the larger
// term is zero).  Out: hi + lo.
template <bool DW>
LG_CRF_DEV void crf_log_dw(float uh, float ul, float& hi, float& lo)
{
    int e, j, mb;
    crf_log_fields(crf_bits(uh), e, j, mb);
    const float m = crf_from_bits(mb);
    const float4 T = crf_tab4(lg_crf_log_tab, j);
    const float c = T.x, Lh = T.y, Ll = T.z;
    // e as float: e + 1.5 2^23 has the bits 0x4b400000 + e
    const float ef = crf_sub(crf_from_bits(0x4b400000 + e), 0x1.8p23f);
    const float ph = crf_mul(m, c);
    const float pl = crf_fma(m, c, crf_neg(ph));
    float rh = crf_sub(ph, 1.0f);  // exact
    float rl;
    if (DW) {
        // + m_lo c, then renormalise (two-sum: m_lo can exceed rh)
        const float ml = crf_mul(ul, crf_from_bits(crf_pow2_bits(-e)));  // exact: ul 2^-e
        const float q = crf_fma(ml, c, pl);
        const float s = crf_add(rh, q);
        const float bb = crf_sub(s, rh);
        rl = crf_add(crf_sub(rh, crf_sub(s, bb)), crf_sub(q, bb));
        rh = s;
    } else {
        // renormalise: pl (up to 2^-25) would otherwise dominate the
        // rounding errors of small r (fast two-sum: rh = 0 or |rh| >= 2^-24)
        const float s = crf_add(rh, pl);
        rl = crf_sub(pl, crf_sub(s, rh));
        rh = s;
    }
    float vh, vl;
    crf_log1p_dw(rh, rl, vh, vl);
    const float a1 = crf_mul(ef, LG_CRF_LN2_HI);
    const float a1l = crf_fma(ef, LG_CRF_LN2_HI, crf_neg(a1));
    const float a1l2 = crf_mul(ef, LG_CRF_LN2_LO);
    const float s1 = crf_add(a1, Lh);
    const float e1 = crf_sub(Lh, crf_sub(s1, a1));
    hi = crf_add(s1, vh);
    const float e2 = crf_sub(vh, crf_sub(hi, s1));
    lo = crf_add(crf_add(e1, e2), crf_add(crf_add(a1l, a1l2), crf_add(Ll, vl)));
}

LG_CRF_DEV float crf_full_log(float x)
{
    float hi, lo, z1, z2;
    crf_log_dw<false>(x, x, hi, lo);
    crf_ziv(hi, lo, z1, z2);
    // normal, positive, finite x with the rounding decided; zero, negative,
    // subnormal, infinite and NaN x in double
    return x >= 0x1p-126f && x <= 0x1.fffffep127f && z1 == z2 ? z1 : crf_slow_log(x);
}

// --------------------------------------------------------------------- atan --
// a = |z|; t = a, or 1/a (as rcp(a) plus one Newton correction, a double
// word) for a > 1.  With t_j = j/512 nearest t, atan t = atan t_j +
// atan(delta), delta = (t - t_j) / (1 + t t_j) as a double word (numerator
// exact by Sterbenz; denominator 1 + t t_j from an exact product; quotient
// from rcp plus one correction step), |delta| <= 2^-10, atan(delta) = delta
// + delta^3 (-1/3 + delta^2/5), truncation delta^7/7 (relative 2^-62), the
// cubic term in float (relative to delta 2^-44).  For a > 1 the result is
// pi/2 - that.  Error about 2^-44.
// atan t for t = th + tl in [0, 1] (tl a few ulp of th at most) as s1 + lo.
LG_CRF_DEV void crf_atan_core(float th, float tl, float& s1, float& lo)
{
    const float S = 0x1.8p23f;
    const float big = crf_fma(th, 512.0f, S);
    const float tj = crf_mul(crf_sub(big, S), 0x1p-9f);
    int j = crf_bits(big) - 0x4b400000;
    j = j < 0 ? 0 : (j > 512 ? 512 : j);  // (in range for every finite t in [0, 1])
    const float2 A = crf_tab2(lg_crf_q_tab + LG_CRF_Q_ATAN, j);
    const float Ah = A.x, Al = A.y;
    const float nh = crf_sub(th, tj);  // exact
    const float qh = crf_mul(th, tj);
    const float ql = crf_fma(th, tj, crf_neg(qh));
    const float dh = crf_add(1.0f, qh);  // 1 >= qh: fast two-sum
    const float dl = crf_add(crf_sub(qh, crf_sub(dh, 1.0f)), crf_fma(tl, tj, ql));
    const float rd = crf_rcp(dh);  // dh in [1, 2]
    const float d0 = crf_mul(nh, rd);
    const float res = crf_add(crf_fma(crf_neg(d0), dh, nh), crf_fma(crf_neg(d0), dl, tl));
    const float d1 = crf_mul(res, rd);
    const float s = crf_mul(d0, d0);
    const float P = crf_fma(s, 0x1.99999ap-3f, -0x1.555556p-2f);
    const float cub = crf_mul(crf_mul(s, d0), P);
    s1 = crf_add(Ah, d0);  // |atan t_j| >= |delta| or t_j = 0
    const float e1 = crf_sub(d0, crf_sub(s1, Ah));
    lo = crf_add(crf_add(e1, Al), crf_add(d1, cub));
}

LG_CRF_DEV float crf_full_atan(float z)
{
    const float a = crf_abs(z);
    const bool inv = a > 1.0f;
    float th = a, tl = 0.0f;
    if (inv) {  // 1/a (a > 2^126 flushes to 0; atan is then RN(pi/2))
        th = crf_rcp(a);
        tl = crf_mul(crf_fma(crf_neg(th), a, 1.0f), th);
    }
    float hi, lo, z1, z2;
    crf_atan_core(th, tl, hi, lo);
    if (inv) {  // pi/2 - (hi + lo)
        const float ph = crf_sub(LG_CRF_PIO2_HI, hi);
        const float pe = crf_sub(crf_sub(LG_CRF_PIO2_HI, ph), hi);
        lo = crf_add(pe, crf_sub(LG_CRF_PIO2_LO, lo));
        hi = ph;
    }
    crf_ziv(hi, lo, z1, z2);
    // finite z with the rounding decided; infinite and NaN z in double.  The
    // sign of z on |result| (z = +-0 gives +-0: the result is 0 there).
    return a <= 0x1.fffffep127f && z1 == z2 ? crf_copysignf(z1, z) : crf_slow_atan(z);
}

// -------------------------------------------------------------------- atanh --
// atanh v = sign(v) atanh(a), a = |v| < 1, by two formulas:
//  * a <= 0.9: with t_j = j/512 nearest a, atanh a = atanh t_j +
//    atanh(delta), delta = (a - t_j) / (1 - a t_j) as a double word
//    (numerator exact; denominator from an exact product and a fast
//    two-sum, at least 0.19; quotient from rcp plus one correction step),
//    |delta| <= 2^-7.6, atanh(delta) = delta + delta^3 (1/3 + delta^2/5),
//    truncation delta^7/7 (relative 2^-48), the cubic term in float;
//    table pairs atanh t_j (2^-48).  Error about 2^-45;
//  * a > 0.9: ln(1 + w) / 2 with w = 2a / (1 - a) as a double word (1 - a
//    exact by a fast two-sum, the quotient from rcp plus one correction
//    step), 1 + w as a two-sum, then the double-word logarithm: 1 + w
//    carries about 2^-49 absolute error, 2^-46 of the result here.
// The SIE family's arguments stay below sqrt(1 - q^2), so its rays take the
// first formula unless q < 0.44.
LG_CRF_DEV float crf_full_atanh(float v)
{
    const float a = crf_abs(v);
    const float one = 1.0f;
    float hi, lo, z1, z2;
    if (a <= 0.9f) {
        const float S = 0x1.8p23f;
        const float big = crf_fma(a, 512.0f, S);
        const float tj = crf_mul(crf_sub(big, S), 0x1p-9f);
        const float2 A = crf_tab2(lg_crf_q_tab + LG_CRF_Q_ATANH, crf_bits(big) - 0x4b400000);
        const float Ah = A.x, Al = A.y;
        const float nh = crf_sub(a, tj);  // exact
        const float qh = crf_mul(a, tj);
        const float ql = crf_fma(a, tj, crf_neg(qh));
        const float dh = crf_sub(one, qh);  // 1 >= qh: fast two-sum
        const float dl = crf_sub(crf_sub(crf_sub(one, dh), qh), ql);
        const float rd = crf_rcp(dh);  // dh in [0.19, 1]
        const float d0 = crf_mul(nh, rd);
        const float res = crf_fma(crf_neg(d0), dl, crf_fma(crf_neg(d0), dh, nh));
        const float d1 = crf_mul(res, rd);
        const float s = crf_mul(d0, d0);
        const float P = crf_fma(s, 0x1.99999ap-3f, 0x1.555556p-2f);
        const float cub = crf_mul(crf_mul(s, d0), P);
        hi = crf_add(Ah, d0);  // |atanh t_j| >= |delta| or t_j = 0: fast two-sum
        const float e1 = crf_sub(d0, crf_sub(hi, Ah));
        lo = crf_add(crf_add(e1, Al), crf_add(d1, cub));
    } else {
        const float dh = crf_sub(one, a);
        const float dl = crf_sub(crf_sub(one, dh), a);  // exact (1 >= a)
        const float n = crf_add(a, a);
        const float rd = crf_rcp(dh);  // dh >= 2^-24
        const float w0 = crf_mul(n, rd);
        const float res = crf_fma(crf_neg(w0), dl, crf_fma(crf_neg(w0), dh, n));
        const float w1 = crf_mul(res, rd);
        // 1 + w0 (two-sum: w0 may exceed 1), + w1
        const float uh = crf_add(one, w0);
        const float bb = crf_sub(uh, one);
        const float ul = crf_add(crf_add(crf_sub(one, crf_sub(uh, bb)), crf_sub(w0, bb)), w1);
        crf_log_dw<true>(uh, ul, hi, lo);
        hi = crf_mul(hi, 0.5f);
        lo = crf_mul(lo, 0.5f);
    }
    crf_ziv(hi, lo, z1, z2);
    // |v| < 1 with the rounding decided; |v| >= 1 and NaN v in double.  The
    // sign of v on |result| (v = +-0 gives +-0).
    return a < 1.0f && z1 == z2 ? crf_copysignf(z1, v) : crf_slow_atanh(v);
}

#ifndef LG_CRF_NO_QUICK
// ------------------------------------------------------------ quick phases --
// exp, log, atan and atanh as the exact render calls them: a first phase of
// 16-24 operations whose error is far below half a float ulp, Ziv's test on
// its interval, and the functions above (out of line) for the lanes it
// leaves undecided.  All F operations run on both lanes of a pair at once.
//
// products that enter only fmas, or sums where the unrounded product serves
// as well: on pairs the packed multiply, which the assembler may contract
// into a following packed add.  (atanh's d, added to a table value, is such a
// product: what its sum loses is taken against the rounded d.  atan's is not,
// there the error term of the sum adds the product itself.)
LG_CRF_DEV float crf_mulx(float a, float b) { return crf_mul(a, b); }
#ifndef LG_CRF_HOST
LG_CRF_DEV float2 crf_mulx(float2 a, float2 b) { return __fmul2_rn(a, b); }
#endif
#ifndef LG_CRF_REST_COUNT
#define LG_CRF_REST_COUNT()
#endif
LG_CRF_COLD float crf_rest_exp(float x) { LG_CRF_REST_COUNT(); return x <= LG_CRF_EXP_ZERO ? 0.0f : crf_full_exp(x); }
LG_CRF_COLD float crf_rest_log(float x) { LG_CRF_REST_COUNT(); return crf_full_log(x); }
LG_CRF_COLD float crf_rest_atan(float x) { LG_CRF_REST_COUNT(); return crf_full_atan(x); }
LG_CRF_COLD float crf_rest_atanh(float x) { LG_CRF_REST_COUNT(); return crf_full_atanh(x); }

// integer fields, in inline PTX as above:
//   exp: z 2^m for k = 1024 m + j, big's bits = bits(1.5 2^23) + k (the
//        constant's bits leave the word in the shift)
//   log: the mantissa in [1, 2) and the sign and biased exponent (times 2^23)
#ifdef LG_CRF_HOST
LG_CRF_DEV int crf_qexp_scale(int zbits, int bits) { return (int)((unsigned)zbits + ((unsigned)(bits & ~1023) << 13)); }
LG_CRF_DEV void crf_qlog_fields(int b, int& mb, int& te)
{
    mb = (b & 0x007fffff) | 0x3f800000;
    te = b & (int)0xff800000;
}
#else
LG_CRF_DEV int crf_qexp_scale(int zbits, int bits)
{
    int r;
    asm("{\n.reg .s32 t;\nand.b32 t, %2, 0xfffffc00;\nshl.b32 t, t, 13;\nadd.s32 %0, %1, t;\n}"
        : "=r"(r)
        : "r"(zbits), "r"(bits));
    return r;
}
LG_CRF_DEV void crf_qlog_fields(int b, int& mb, int& te)
{
    asm("{\n.reg .b32 t;\nand.b32 t, %2, 0x007fffff;\nor.b32 %0, t, 0x3f800000;\nand.b32 %1, %2, 0xff800000;\n}"
        : "=r"(mb), "=r"(te)
        : "r"(b));
}
#endif

#define LG_CRF_QEXP_REM (0x1.ap-34f - 0x1p-24f)
// e^x, |x| <= 87: x = k ln2/1024 + r, |r| <= 2^-11.5, k - 1 = 1024 m + j; with
// T = 2^((j + 1)/1024) = th + tl in (1, 2], e^x 2^-m = th + (th rh + (th (rl + rh (rh/2 + rl)) + tl
// + tl rh)): rh = x - k L_hi exact, rl = -k L_lo.  Absolute error of the sum before its
// rounding: that of the inner sum (2^-35), r^3/6 (2^-36.2 with T < 2), the
// rest below 2^-41; the table's second entry holds tl + D with D = 1.625
// 2^-35, the interval's half-width, so z = th + c rounds its upper end.  th +
// c - 2D rounds to z too if the exact remainder of that sum, c - (z - th), is at
// least 2D - 2^-24: z is above 1 (why k - 1), so half an ulp below it is 2^-24
// at least.
template <class F>
LG_CRF_DEV F lg_crf_exp(F x)
{
    const F big = crf_fma(x, crf_bc<F>(LG_CRF_QEXP_INVL), crf_bc<F>(0x1.7ffffep23f));
    const F kf = crf_add(big, crf_bc<F>(-0x1.7ffffep23f));
    const F rh = crf_fma(kf, crf_bc<F>(-LG_CRF_QEXP_LHI), x);
    const F rl = crf_mulx(kf, crf_bc<F>(-LG_CRF_QEXP_LLO));
    const F sm = crf_fma(rh, crf_fma(rh, crf_bc<F>(0.5f), rl), rl);
    F th, tl;
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) {
        const float2 T = crf_qtab(LG_CRF_Q_EXP, (unsigned)(crf_bits(crf_get(big, i)) & 1023) * 8u);
        crf_set(th, i, T.x);
        crf_set(tl, i, T.y);
    }
    const F c = crf_fma(th, rh, crf_fma(th, sm, crf_fma(tl, rh, tl)));
    const F z = crf_add(th, c);
    const F rem = crf_sub(c, crf_sub(z, th));
    F out;
    bool ok[2];
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) {
        ok[i] = crf_fabsf(crf_get(x, i)) <= 87.0f && crf_get(rem, i) >= LG_CRF_QEXP_REM;
        crf_set(out, i, crf_from_bits(crf_qexp_scale(crf_bits(crf_get(z, i)), crf_bits(crf_get(big, i)))));
    }
    if (!crf_all<F>(ok)) {
        bool zero[2];  // the wings of compact profiles
#pragma unroll
        for (int i = 0; i < crf_lanes<F>::n; ++i) zero[i] = crf_get(x, i) <= LG_CRF_EXP_ZERO;
        if (crf_all<F>(zero)) return crf_bc<F>(0.0f);
#pragma unroll
        for (int i = 0; i < crf_lanes<F>::n; ++i)
            if (!ok[i]) crf_set(out, i, crf_rest_exp(crf_get(x, i)));
    }
    return out;
}

// ln x, 2^-90 <= x < 2^91: x = 2^e m, m in [1, 2), c = 1/m cut to 11
// significant bits (from the reciprocal estimate; any estimate serves), so that
// r = m c - 1 (|r| <= 2^-10) is exact; ln x = ((e - 1/2) ln2_hi + Lh) + (r + (r^2
// (r/3 - 1/2) + (e - 1/2) ln2_lo + Ll)) with ln2/2 - ln c = Lh + Ll, ln2_hi a
// multiple of 2^-17 and Lh of 2^-18: the first sum is exact.  (The half centres
// the exponents that one comparison of |e - 1/2| then admits; zero, subnormal,
// negative, infinite and NaN x fail it.)  Absolute error: the sum with r (2^-34
// at most), (e - 1/2) ln2_lo + Ll (2^-36), r^4/4 (2^-42); the table's Ll holds
// D = 1.375 2^-34 more, and the interval's lower end is 3.75 2^-34 below, its
// own rounding included.  Results near 0 are left to the full phase.
// Out: s1, r and t with ln x + D = s1 + (r + t), and e - 1/2 (times 2^23).
template <class F>
LG_CRF_DEV void crf_quick_log(F x, F& s1, F& r, F& t, F& e)
{
    F m, c, Lh, Ll, ef;
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) {
        int mb, te;
        crf_qlog_fields(crf_bits(crf_get(x, i)), mb, te);
        const int cb = crf_bits(crf_rcp(crf_from_bits(mb))) & (int)0xffffe000;
        const float2 T = crf_qtab(LG_CRF_Q_LOG, ((unsigned)cb >> 10) - (0x3effe000u >> 10));
        crf_set(m, i, crf_from_bits(mb));
        crf_set(c, i, crf_from_bits(cb));
        crf_set(Lh, i, T.x);
        crf_set(Ll, i, T.y);
        crf_set(ef, i, (float)te);  // exact
    }
    r = crf_fma(m, c, crf_bc<F>(-1.0f));
    e = crf_add(ef, crf_bc<F>(-127.5f * 0x1p23f));
    s1 = crf_fma(e, crf_bc<F>(LG_CRF_QLN2_HI), Lh);
    const F lo = crf_fma(e, crf_bc<F>(LG_CRF_QLN2_LO), Ll);
    const F w = crf_fma(r, crf_bc<F>(0x1.555556p-2f), crf_bc<F>(-0.5f));
    t = crf_fma(crf_mulx(r, r), w, lo);
}
#define LG_CRF_QLOG_E (90.5f * 0x1p23f)
template <class F>
LG_CRF_DEV F lg_crf_log(F x)
{
    F s1, r, t, e;
    crf_quick_log(x, s1, r, t, e);
    const F a = crf_add(r, t);
    F out = crf_add(s1, a);
    const F z2 = crf_add(s1, crf_add(a, crf_bc<F>(-0x1.ep-33f)));
    bool ok[2];
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i)
        ok[i] = crf_fabsf(crf_get(e, i)) <= LG_CRF_QLOG_E && crf_get(out, i) == crf_get(z2, i);
    if (!crf_all<F>(ok)) {
#pragma unroll
        for (int i = 0; i < crf_lanes<F>::n; ++i)
            if (!ok[i]) crf_set(out, i, crf_rest_log(crf_get(x, i)));
    }
    return out;
}

// both ends of the interval hi + lo -+ |hi| 2^-38, rounded
template <class F>
LG_CRF_DEV void crf_quick_ziv(F hi, F lo, F& z1, F& z2)
{
    z1 = crf_add(hi, crf_fma(hi, crf_bc<F>(0x1p-38f), lo));
    z2 = crf_add(hi, crf_fma(hi, crf_bc<F>(-0x1p-38f), lo));
}

// atan t for t in [0, 2] (callers keep every t, NaN included, in that range:
// it indexes the table): with t_j = j/512 nearest t, n = t - t_j and d = n /
// (1 + t_j^2) (the denominator exact), atan t = atan t_j + d - t_j d^2 + (t_j^2
// - 1/3) d^3 + O(d^4 t_j) (Taylor's series in d; |d| <= 2^-10, the omitted
// term 2^-40 of the result).  d as a double word from the reciprocal estimate
// and one correction.  The series' signs are kept negated (nd = -d) so that
// no operand needs a negation.
template <class F, bool DW>
LG_CRF_DEV void crf_quick_atan(F t, F tl, F& s1, F& lo)
{
    const F big = crf_add(t, crf_bc<F>(0x1.8p14f));  // t to the nearest 2^-9
    const F tj = crf_add(big, crf_bc<F>(-0x1.8p14f));
    F Ah, Al, nr;
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) {
        const float2 A = crf_qtab(LG_CRF_Q_ATAN, (unsigned)(crf_bits(crf_get(big, i)) - 0x46c00000) * 8u);
        crf_set(Ah, i, A.x);
        crf_set(Al, i, A.y);
    }
    const F n = crf_fma(tj, crf_bc<F>(-1.0f), t);
    const F s = crf_fma(tj, tj, crf_bc<F>(1.0f));
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) crf_set(nr, i, crf_rcp(-crf_get(s, i)));
    const F nd = crf_mul(n, nr);  // rounded: its error is in res, so ne below has to take the same value
    F res = crf_fma(nd, s, n);
    if (DW) res = crf_add(res, tl);
    F nd1 = crf_mulx(res, nr);
    if (DW) nd1 = crf_fma(crf_add(nd1, nd1), crf_mulx(tj, nd), nd1);  // the square's cross term with tl
    F K = crf_add(s, crf_bc<F>(-0x1.555556p+0f));
    if (DW) K = crf_fma(crf_mulx(tj, crf_add(s, crf_bc<F>(-2.0f))), nd, K);  // the fourth power's term
    const F P = crf_fma(K, nd, tj);
    const F nc = crf_fma(crf_mulx(nd, nd), P, nd1);
    s1 = crf_fma(nd, crf_bc<F>(-1.0f), Ah);
    const F ne = crf_add(nd, crf_fma(Ah, crf_bc<F>(-1.0f), s1));
    lo = crf_fma(crf_add(ne, nc), crf_bc<F>(-1.0f), Al);
}
// pairs with a lane above 2 (or NaN): t = 1/a in lanes above 1 as a double word (a >
// 2^126 flushes it to 0: the result is RN(pi/2)), and pi/2 - atan t
template <class F>
LG_CRF_COLD F crf_wide_atan(F z)
{
    const F a = crf_abs(z);
    F r0, th, tl, s1, lo, z1, z2, out;
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) crf_set(r0, i, crf_get(a, i) > 1.0f ? crf_rcp(crf_get(a, i)) : 1.0f);
    const F r1 = crf_mulx(crf_fma(crf_neg(r0), a, crf_bc<F>(1.0f)), r0);
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) {
        const bool inv = crf_get(a, i) > 1.0f;
        // (NaN takes 1 here and the double evaluation below)
        crf_set(th, i, inv || !(crf_get(a, i) <= 1.0f) ? crf_get(r0, i) : crf_get(a, i));
        crf_set(tl, i, inv ? crf_get(r1, i) : 0.0f);
    }
    crf_quick_atan<F, true>(th, tl, s1, lo);
    const F ph = crf_fma(s1, crf_bc<F>(-1.0f), crf_bc<F>(LG_CRF_PIO2_HI));
    const F pe = crf_sub(crf_sub(crf_bc<F>(LG_CRF_PIO2_HI), ph), s1);
    const F pl = crf_add(pe, crf_sub(crf_bc<F>(LG_CRF_PIO2_LO), lo));
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i)
        if (crf_get(a, i) > 1.0f) {
            crf_set(s1, i, crf_get(ph, i));
            crf_set(lo, i, crf_get(pl, i));
        }
    crf_quick_ziv(s1, lo, z1, z2);
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) {
        const float zi = crf_get(z, i);
        const bool ok = crf_fabsf(zi) <= 0x1.fffffep127f && crf_get(z1, i) == crf_get(z2, i);
        crf_set(out, i, ok ? crf_copysignf(crf_get(z1, i), zi) : crf_rest_atan(zi));
    }
    return out;
}
template <class F>
LG_CRF_DEV F lg_crf_atan(F z)
{
    const F a = crf_abs(z);
    bool in = true;
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) in = in && crf_get(a, i) <= 2.0f;  // (SIE: axis ratios from 0.45)
    if (!in) return crf_wide_atan(z);
    F s1, lo, z1, z2, out;
    crf_quick_atan<F, false>(a, a, s1, lo);
    crf_quick_ziv(s1, lo, z1, z2);
    bool ok[2];
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) {
        ok[i] = crf_get(z1, i) == crf_get(z2, i);
        crf_set(out, i, crf_copysignf(crf_get(z1, i), crf_get(z, i)));
    }
    if (!crf_all<F>(ok)) {
#pragma unroll
        for (int i = 0; i < crf_lanes<F>::n; ++i)
            if (!ok[i]) crf_set(out, i, crf_rest_atan(crf_get(z, i)));
    }
    return out;
}

// atanh v, a = |v| <= 0.9: with t_j = j/512 nearest a and n = a - t_j, atanh a =
// atanh t_j + atanh d, d = n / (1 - a t_j), 1 - a t_j = (1 - t_j^2) - n t_j as a
// double word (both terms exact), d as a double word from the reciprocal
// estimate and one correction, atanh d = d + d^3/3 (|d| <= 2^-7.6 at a = 0.9:
// d^5/5 is 2^-40.8 of the result).
template <class F>
LG_CRF_DEV F lg_crf_atanh(F v)
{
    const F a = crf_abs(v);
    const F big = crf_add(a, crf_bc<F>(0x1.8p14f));
    const F tj = crf_add(big, crf_bc<F>(-0x1.8p14f));
    F Ah, Al, rd;
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) {
        // (the mask keeps arguments outside the range inside the table)
        const float2 A = crf_qtab(LG_CRF_Q_ATANH, (unsigned)(crf_bits(crf_get(big, i)) & 511) * 8u);
        crf_set(Ah, i, A.x);
        crf_set(Al, i, A.y);
    }
    const F n = crf_fma(tj, crf_bc<F>(-1.0f), a);
    const F nD = crf_fma(tj, tj, crf_bc<F>(-1.0f));
    const F nh = crf_fma(n, tj, nD);
    const F nl = crf_fma(n, tj, crf_fma(nh, crf_bc<F>(-1.0f), nD));
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) crf_set(rd, i, crf_rcp(-crf_get(nh, i)));
    const F d = crf_mulx(n, rd);
    const F d1 = crf_mulx(crf_fma(d, nl, crf_fma(d, nh, n)), rd);
    const F c = crf_fma(crf_mulx(crf_mulx(d, d), d), crf_bc<F>(0x1.555556p-2f), d1);
    const F s1 = crf_add(Ah, d);
    const F ne = crf_fma(d, crf_bc<F>(-1.0f), crf_fma(Ah, crf_bc<F>(-1.0f), s1));
    const F lo = crf_add(crf_fma(ne, crf_bc<F>(-1.0f), c), Al);
    F z1, z2;
    crf_quick_ziv(s1, lo, z1, z2);
    F out;
    bool ok[2];
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) {
        ok[i] = crf_get(a, i) <= 0.9f && crf_get(z1, i) == crf_get(z2, i);
        crf_set(out, i, crf_copysignf(crf_get(z1, i), crf_get(v, i)));
    }
    if (!crf_all<F>(ok)) {
#pragma unroll
        for (int i = 0; i < crf_lanes<F>::n; ++i)
            if (!ok[i]) crf_set(out, i, crf_rest_atanh(crf_get(v, i)));
    }
    return out;
}
#endif  // LG_CRF_NO_QUICK

// ------------------------------------------------- sincos, pow, atan2 (scalar) --
// The EPL lens's functions, one value at a time: for scalar calls, and for
// the lanes that the quick phases of pairs (below) leave undecided.

LG_CRF_DEV void crf_two_sum(float a, float b, float& s, float& e)
{
    s = crf_add(a, b);
    const float bb = crf_sub(s, a);
    e = crf_add(crf_sub(a, crf_sub(s, bb)), crf_sub(b, bb));
}

// Ziv's test with the margin |hi| 2^-40 + floor (floor: an absolute error
// bound of results near zero); z the rounded result when it holds
LG_CRF_DEV bool crf_ziv1(float hi, float lo, float floor_, float& z)
{
    const float m = crf_fma(crf_fabsf(hi), LG_CRF_ZIV, floor_);
    const float z1 = crf_add(hi, crf_add(lo, m)), z2 = crf_add(hi, crf_sub(lo, m));
    z = z1;
    return z1 == z2;
}

// sin x and cos x.  x = k pi/2 + r with k = rint(x 2/pi) (|x| <= 128, so
// |k| < 2^7) and r = ((x - k P1) - k P2) - k P3 as a double word: k P1 and
// k P2 exact (P1, P2 of 17 significant bits), the first difference exact by
// Sterbenz, the second by a two-sum, pi/2 - P1 - P2 - P3 below 2^-59, so
// |error| <= 2^-51 (none for k = 0).  r = a + s with a = j/256 nearest r
// (s exact, |s| <= 2^-9): sin r = sin a cos s + cos a sin s, cos r = cos a
// cos s - sin a sin s with sin a, cos a as table pairs (2^-48), sin s = s -
// s^3/6 + s^5/120 (truncation 2^-65), cos s - 1 = -s^2/2 + s^4/24 - s^6/720
// with s^2 exact; the leading products exact (fma), the sums by two-sums.
// Relative error about 2^-46 plus the reduction's 2^-51 absolute: the
// rounding test takes an absolute floor of 2^-46 when k != 0.  |x| > 128,
// infinite and NaN x, and undecided roundings in double.
LG_CRF_DEV void lg_crf_sincos(float x, float* sp, float* cp)
{
    const bool inr = crf_fabsf(x) <= 128.0f;
    const float xr = inr ? x : 0.0f;
    const float S = 0x1.8p23f;
    const float big = crf_fma(xr, LG_CRF_INV_PIO2, S);
    const float kf = crf_sub(big, S);
    const int k = crf_bits(big) - 0x4b400000;
    const float r1 = crf_fma(-kf, LG_CRF_PIO2_1, xr);  // exact
    float rh, e;
    crf_two_sum(r1, crf_mul(-kf, LG_CRF_PIO2_2), rh, e);
    const float rl = crf_fma(-kf, LG_CRF_PIO2_3, e);
    const float bj = crf_fma(rh, 256.0f, S);
    const int j = crf_bits(bj) - 0x4b400000;  // |j| <= 201
    const float a = crf_mul(crf_sub(bj, S), 0x1p-8f);
    const float s0 = crf_sub(rh, a);  // exact
    const float4 T = crf_tab4(lg_crf_sc_tab, (j + 201));
    const float sah = T.x, sal = T.y, cah = T.z, cal = T.w;
    // sin s = s0 + Sl; cos s - 1 = Ch + Cl
    const float s2 = crf_mul(s0, s0);
    const float s2l = crf_fma(crf_add(s0, s0), rl, crf_fma(s0, s0, -s2));
    const float Sl = crf_fma(crf_mul(s2, s0), crf_fma(s2, 0x1.111112p-7f, -0x1.555556p-3f), rl);
    const float Ch = crf_mul(s2, -0.5f);  // exact
    const float Cl = crf_fma(crf_mul(s2, s2), crf_fma(s2, -0x1.6c16c2p-10f, 0x1.555556p-5f), crf_mul(s2l, -0.5f));
    // sin r = sa + ca s0 + sa Ch + (sa Cl + ca Sl + cal s0 + sal)
    const float p1 = crf_mul(cah, s0), e1 = crf_fma(cah, s0, -p1);
    const float p2 = crf_mul(sah, Ch), e2 = crf_fma(sah, Ch, -p2);
    float u, eu;
    crf_two_sum(sah, p1, u, eu);
    const float sh = crf_add(u, p2);  // |u| >= |p2|: fast two-sum
    const float ev = crf_sub(p2, crf_sub(sh, u));
    const float sl = crf_add(crf_add(ev, eu),
                             crf_add(crf_add(e1, e2), crf_fma(sah, Cl, crf_fma(cah, Sl, crf_fma(cal, s0, sal)))));
    // cos r = ca - sa s0 + ca Ch + (ca Cl - sa Sl - sal s0 + cal)
    const float p3 = crf_mul(sah, s0), e3 = crf_fma(sah, s0, -p3);
    const float p4 = crf_mul(cah, Ch), e4 = crf_fma(cah, Ch, -p4);
    float u2, eu2;
    crf_two_sum(cah, -p3, u2, eu2);
    const float ch = crf_add(u2, p4);  // |u2| >= 1/2 >= |p4|: fast two-sum
    const float ev2 = crf_sub(p4, crf_sub(ch, u2));
    const float cl = crf_add(crf_add(ev2, eu2),
                             crf_add(crf_sub(e4, e3), crf_fma(cah, Cl, crf_fma(-sah, Sl, crf_fma(-sal, s0, cal)))));
    // quadrant: sin x = (sin r, cos r, -sin r, -cos r)[k & 3], cos x = (cos r,
    // -sin r, -cos r, sin r)[k & 3]
    const int q = k & 3;
    const bool swap = q & 1, sneg = q >= 2, cneg = q == 1 || q == 2;
    float xsh = swap ? ch : sh, xsl = swap ? cl : sl, xch = swap ? sh : ch, xcl = swap ? sl : cl;
    if (sneg) {
        xsh = -xsh;
        xsl = -xsl;
    }
    if (cneg) {
        xch = -xch;
        xcl = -xcl;
    }
    const float fl = k != 0 ? 0x1p-46f : 0.0f;
    float zs, zc;
    const bool oks = crf_ziv1(xsh, xsl, fl, zs) && inr, okc = crf_ziv1(xch, xcl, fl, zc) && inr;
    *sp = oks ? (x == 0.0f ? x : zs) : crf_slow_sin(x);  // (sin of -0 is -0)
    *cp = okc ? zc : crf_slow_cos(x);
}

// x^y = e^(y ln x): ln x as a double word (crf_log_dw, relative error below
// 2^-42), t = y ln x as a double word (the product exact by an fma), e^t
// from the exp tail with the low part of t added to the reduced argument by
// a two-sum.  Relative error below about |t| 2^-42 + 2^-42, so the rounding
// test's margin grows with |t|.  Positive normal x with t in [-87, 88] (a
// normal result) and the rounding decided; everything else in double.
LG_CRF_DEV float lg_crf_pow(float x, float y)
{
    const bool xin = x >= 0x1p-126f && x <= 0x1.fffffep127f;
    const float xr = xin ? x : 1.0f;
    float lh, ll;
    crf_log_dw<false>(xr, xr, lh, ll);
    const float th = crf_mul(y, lh);
    const float tl = crf_fma(y, ll, crf_fma(y, lh, -th));
    const bool tin = th >= -87.0f && th <= 88.0f;  // (false for NaN)
    const float t = tin ? th : 0.0f, tlo = tin ? tl : 0.0f;
    const float S = 0x1.8p23f;
    const float big = crf_fma(t, LG_CRF_EXP_INVL, S);
    const float kf = crf_sub(big, S);
    const float r0 = crf_fma(-kf, LG_CRF_EXP_LHI, t);  // exact
    float rh, e;
    crf_two_sum(r0, tlo, rh, e);
    const float rl = crf_fma(-kf, LG_CRF_EXP_LLO, e);
    float yh, yl;
    int m;
    crf_exp_tail(big, rh, rl, yh, yl, m);
    const float mrel = crf_fma(crf_fabsf(t), 0x1p-41f, LG_CRF_ZIV);
    const float mg = crf_mul(crf_fabsf(yh), mrel);
    const float z1 = crf_add(yh, crf_add(yl, mg)), z2 = crf_add(yh, crf_sub(yl, mg));
    if (xin && tin && z1 == z2) return crf_from_bits(crf_add_exp(crf_bits(z1), m));
    return crf_slow_pow(x, y);
}

// atan2(y, x): q = min(|x|, |y|) / max(|x|, |y|) in [0, 1] as a double word
// (rcp plus one correction step, relative error 2^-46), atan q from the atan
// core, then pi/2 - that where |y| > |x| and pi - that where x < 0 (double-
// word constants; fast two-sums, the constant being the larger), the sign
// of y.  Relative error about 2^-44.  min(|x|, |y|) >= 2^-100, max(|x|, |y|)
// < 2^126, a quotient above 2^-100 (so the result is normal) and the
// rounding decided; zeros, infinities, NaN, tiny or huge arguments and the
// rest in double.
LG_CRF_DEV float lg_crf_atan2(float y, float x)
{
    const float ax = crf_fabsf(x), ay = crf_fabsf(y);
    const bool swap = ay > ax;
    float num = swap ? ax : ay, den = swap ? ay : ax;
    // the quotient's remainder exact (no underflow: num >= 2^-100), the
    // reciprocal normal (den < 2^126) and the quotient above 2^-100
    const bool in = den < 0x1p126f && num >= 0x1p-100f && num >= crf_mul(den, 0x1p-100f);
    if (!in) {
        num = 1.0f;
        den = 1.0f;
    }
    const float rd = crf_rcp(den);
    const float q0 = crf_mul(num, rd);
    const float res = crf_fma(-q0, den, num);  // exact
    const float q1 = crf_mul(res, rd);
    float s1, lo;
    crf_atan_core(q0, q1, s1, lo);
    float hi = s1;
    if (swap) {  // pi/2 - (s1 + lo)
        const float ph = crf_sub(LG_CRF_PIO2_HI, s1);
        const float pe = crf_sub(crf_sub(LG_CRF_PIO2_HI, ph), s1);
        lo = crf_add(pe, crf_sub(LG_CRF_PIO2_LO, lo));
        hi = ph;
    }
    if (x < 0.0f) {  // pi - (hi + lo)
        const float PIH = crf_mul(LG_CRF_PIO2_HI, 2.0f), PIL = crf_mul(LG_CRF_PIO2_LO, 2.0f);
        const float ph = crf_sub(PIH, hi);
        const float pe = crf_sub(crf_sub(PIH, ph), hi);
        lo = crf_add(pe, crf_sub(PIL, lo));
        hi = ph;
    }
    float z;
    if (in && crf_ziv1(hi, lo, 0.0f, z)) return crf_copysignf(z, y);
    return crf_slow_atan2(y, x);
}

#ifndef LG_CRF_NO_QUICK
// ------------------------------------------- quick phases of the EPL lens --
// x^y for one exponent: ln x = s1 + r + t from the quick log, T = y ln x as a
// double word (y s1 exactly, y t and y r added, a two-sum), e^T as in
// lg_crf_exp with the low part added to the reduction's.  Error of T in units
// of 2^-34 |y|: the roundings of (e - 1/2) ln2_lo + Ll, of t, of its shift back
// by D and of y t added to the product's error 1/8 each (t stays below 2^-12.8),
// ln2_lo's own 0.09, the rounding of y r added to that 1.14 (a sum up to 1.14
// 2^-10 |y|); the square of T's low part, which the exp leaves out, 0.14 (2^-37,
// for |T| above 64 only, so |y| above 1): 1.9 in all.  A power is below 2 times
// its exp's scale, so that is 0.95 2^-32 |y|, and the interval of the exp is
// widened by 2^-32 |y| each way.  (r and t summed to a float first were 1
// more.)  x in the log's range with |T| <= 86; the rest, and undecided
// roundings, in the full phase.
LG_CRF_COLD float crf_rest_pow(float x, float y) { LG_CRF_REST_COUNT(); return lg_crf_pow(x, y); }
template <class F>
LG_CRF_DEV F lg_crf_pow1(F x, float y)
{
    F s1, r, t, e;
    crf_quick_log(x, s1, r, t, e);
    const F Y = crf_bc<F>(y);
    const F ph = crf_mul(Y, s1);
    const F pl = crf_fma(Y, r, crf_fma(Y, crf_add(t, crf_bc<F>(-0x1.6p-34f)), crf_fma(Y, s1, crf_neg(ph))));
    const F T = crf_add(ph, pl);  // two-sum
    const F bb = crf_sub(T, ph);
    const F Tl = crf_add(crf_sub(ph, crf_sub(T, bb)), crf_sub(pl, bb));
    const F big = crf_fma(T, crf_bc<F>(LG_CRF_QEXP_INVL), crf_bc<F>(0x1.7ffffep23f));
    const F kf = crf_add(big, crf_bc<F>(-0x1.7ffffep23f));
    const F rh = crf_fma(kf, crf_bc<F>(-LG_CRF_QEXP_LHI), T);
    const F rl = crf_fma(kf, crf_bc<F>(-LG_CRF_QEXP_LLO), Tl);
    const F sm = crf_fma(rh, crf_fma(rh, crf_bc<F>(0.5f), rl), rl);
    F th, tl;
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) {
        const float2 E = crf_qtab(LG_CRF_Q_EXP, (unsigned)(crf_bits(crf_get(big, i)) & 1023) * 8u);
        crf_set(th, i, E.x);
        crf_set(tl, i, E.y);
    }
    const float wide = crf_mul(crf_fabsf(y), 0x1p-32f);
    const F c = crf_fma(th, rh, crf_add(crf_fma(th, sm, crf_fma(tl, rh, tl)), crf_bc<F>(wide)));
    const F z = crf_add(th, c);
    const F rem = crf_sub(c, crf_sub(z, th));
    const float low = crf_fma(wide, 2.0f, LG_CRF_QEXP_REM);
    F out;
    bool ok[2];
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) {
        ok[i] = crf_fabsf(crf_get(e, i)) <= LG_CRF_QLOG_E && crf_fabsf(crf_get(T, i)) <= 86.0f && crf_get(rem, i) >= low;
        crf_set(out, i, crf_from_bits(crf_qexp_scale(crf_bits(crf_get(z, i)), crf_bits(crf_get(big, i)))));
    }
    if (!crf_all<F>(ok)) {
#pragma unroll
        for (int i = 0; i < crf_lanes<F>::n; ++i)
            if (!ok[i]) crf_set(out, i, crf_rest_pow(crf_get(x, i), y));
    }
    return out;
}

// The EPL lens's polar frame of a point (X, Y): r = sqrt(X^2 + Y^2) with
// every operation rounded, phi = atan2(Y, X) rounded, and the sine and
// cosine of that float phi and of 2 phi, each correctly rounded, in one
// computation instead of an atan2 and two sincos:
//  * H = X^2 + Y^2 as a double word (exact products; its high part is the
//    rounded sum r is the root of), 1/sqrt(H) = y0 + y1 from the reciprocal
//    square root estimate and one Newton step, so cos and sin of the exact
//    angle are X and Y times it;
//  * the exact angle from the atan of min/max as in lg_crf_atan, then phi =
//    its rounding, and rem = angle - phi;
//  * sin phi = sin(angle) - rem cos(angle), cos phi likewise (rem^2/2 is
//    below 2^-47), sin 2phi = 2 sin phi cos phi, cos 2phi = +-(1 - 2 m^2) with
//    m the smaller of the two.
// Error bounds for estimates 2^-22 off (the hardware's: 2^-23 and 2^-22.9),
// in units of 2^-42; in brackets the largest error met on 4 10^7 points with
// estimates that far off either way at random:
//  * sqrt(h), relative: the square of g's error, (1.25 2^-22)^2 / 2, and the
//    roundings of h - g^2 and of its product: 0.7 [0.6], margin 4;
//  * 1/sqrt(H), relative: Newton's step 3/8 (2.5 2^-22)^2 = 0.6, the roundings
//    of 1 - g y0 and of what is added to it 0.4, of y1 0.1; with the rounding
//    of their low parts, sin and cos of the angle 1.0;
//  * atan q, relative: q 0.5, the low part of d (up to 2.5 2^-22 of it: three
//    roundings and the estimate) 1.1, its part in the cube, left out, 2.5, the
//    square 0.65, the cube 0.4, the fifth power 0.8, the sums 1.5: 7.8 [4.0],
//    near q = 2^-10; absolute 1.5 [0.6], and 2.1 with the multiple of pi/2.
//    phi has the margin 16 |phi| of crf_quick_ziv;
//  * sin phi: the angle's error times the cosine, the sine's 1.0 and its
//    rounding: 9.3 |phi| [4.0] below |phi| = 0.36, margin 11 |phi|, and above
//    2.7 [0.8], margin 4; cos phi likewise 2.7 [0.8], margin 4;
//  * sin phi cos phi: both of these, the product of the low parts 0.5 and
//    roundings: 12.4 |phi| [4.4] and 4.4 [0.9], margins 13.75 |phi| and 5;
//  * cos 2phi: 4 |m| times m's error 7.2, twice the square of m's low part
//    1.0, roundings 1.0: 9.2 [2.6], margin 10.
// ok[i]: every rounding of lane i decided; its range excludes axes and
// extreme sizes (min/max < 2^-20, H outside [2^-60, 2^60]), which the caller
// sends through the one-value functions.
template <class F>
LG_CRF_DEV void crf_quick_polar(F X, F Y, F& r, F& c, F& s, F& c2, F& s2, bool (&ok)[2])
{
    F den, num, y0, rd;
    bool swap[2];
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) {
        const float ax = crf_fabsf(crf_get(X, i)), ay = crf_fabsf(crf_get(Y, i));
        swap[i] = ay > ax;
        crf_set(den, i, swap[i] ? ay : ax);
        crf_set(num, i, swap[i] ? ax : ay);
    }
    const F A = crf_mul(den, den), B = crf_mul(num, num);
    const F h = crf_add(A, B);
    const F hl = crf_add(crf_sub(B, crf_sub(h, A)), crf_add(crf_fma(den, den, crf_neg(A)), crf_fma(num, num, crf_neg(B))));
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) {
        crf_set(y0, i, crf_rsqrt(crf_get(h, i)));
        crf_set(rd, i, crf_rcp(crf_get(den, i)));
    }
    // r
    const F g = crf_mul(h, y0);
    const F hy = crf_mulx(y0, crf_bc<F>(0.5f));
    const F g1 = crf_mulx(crf_fma(crf_neg(g), g, h), hy);
    r = crf_add(g, crf_fma(g, crf_bc<F>(0x1p-40f), g1));
    const F r2 = crf_add(g, crf_fma(g, crf_bc<F>(-0x1p-40f), g1));
    // 1/sqrt(H) = y0 + y1; cos, sin of the exact angle
    const F pe = crf_fma(hl, y0, crf_fma(h, y0, crf_neg(g)));
    const F y1 = crf_mulx(hy, crf_fma(crf_neg(pe), y0, crf_fma(crf_neg(g), y0, crf_bc<F>(1.0f))));
    const F ch = crf_mul(X, y0), sh = crf_mul(Y, y0);
    F cl = crf_fma(X, y1, crf_fma(X, y0, crf_neg(ch)));
    F sl = crf_fma(Y, y1, crf_fma(Y, y0, crf_neg(sh)));
    // the angle in [0, pi]: B + sg atan(num/den)
    F q0 = crf_mul(num, rd);
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i)  // NaN and infinite quotients (left undecided) stay inside the table
        crf_set(q0, i, crf_get(q0, i) <= 1.0f ? crf_get(q0, i) : 1.0f);
    const F q1 = crf_mulx(crf_fma(crf_neg(q0), den, num), rd);
    F ah, al, Bh, Bl, sg;
    crf_quick_atan<F, true>(q0, q1, ah, al);
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) {
        const bool neg = crf_get(X, i) < 0.0f;
        crf_set(sg, i, swap[i] != neg ? -1.0f : 1.0f);
        crf_set(Bh, i, swap[i] ? LG_CRF_PIO2_HI : (neg ? 2.0f * LG_CRF_PIO2_HI : 0.0f));
        crf_set(Bl, i, swap[i] ? LG_CRF_PIO2_LO : (neg ? 2.0f * LG_CRF_PIO2_LO : 0.0f));
    }
    const F zh = crf_fma(sg, ah, Bh);
    const F zl = crf_fma(sg, al, crf_add(crf_fma(sg, ah, crf_sub(Bh, zh)), Bl));
    F z1, z2;
    crf_quick_ziv(zh, zl, z1, z2);
    // rem = angle - phi, with the sign of Y; sin, cos of phi
    F rem = crf_add(zl, crf_sub(zh, z1));
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i)
        crf_set(rem, i, crf_from_bits(crf_bits(crf_get(rem, i)) ^ (crf_bits(crf_get(Y, i)) & (int)0x80000000)));
    sl = crf_fma(crf_neg(rem), ch, sl);
    cl = crf_fma(rem, sh, cl);
    F ms = crf_mulx(z1, crf_bc<F>(0x1.6p-39f));
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) crf_set(ms, i, crf_get(ms, i) < 0x1p-40f ? crf_get(ms, i) : 0x1p-40f);
    const F mc = crf_bc<F>(0x1p-40f), mk = crf_bc<F>(0x1.4p-39f);
    s = crf_add(sh, crf_add(sl, ms));
    const F sb = crf_add(sh, crf_sub(sl, ms));
    c = crf_add(ch, crf_add(cl, mc));
    const F cb = crf_add(ch, crf_sub(cl, mc));
    // sin 2phi
    const F ph = crf_mul(sh, ch);
    const F pl = crf_fma(sh, cl, crf_fma(sl, ch, crf_fma(sh, ch, crf_neg(ph))));
    s2 = crf_add(ph, crf_fma(ms, crf_bc<F>(1.25f), pl));
    const F s2b = crf_add(ph, crf_fma(ms, crf_bc<F>(-1.25f), pl));
    // cos 2phi
    F mh, ml;
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) {
        crf_set(mh, i, swap[i] ? crf_get(ch, i) : crf_get(sh, i));
        crf_set(ml, i, swap[i] ? crf_get(cl, i) : crf_get(sl, i));
    }
    const F q = crf_mul(mh, mh);
    const F qe = crf_fma(crf_mulx(mh, ml), crf_bc<F>(2.0f), crf_fma(mh, mh, crf_neg(q)));
    const F k = crf_fma(q, crf_bc<F>(-2.0f), crf_bc<F>(1.0f));
    const F ke = crf_fma(qe, crf_bc<F>(-2.0f), crf_fma(q, crf_bc<F>(-2.0f), crf_sub(crf_bc<F>(1.0f), k)));
    const F k1 = crf_add(k, crf_add(ke, mk));
    const F k2 = crf_add(k, crf_sub(ke, mk));
#pragma unroll
    for (int i = 0; i < crf_lanes<F>::n; ++i) {
        crf_set(c2, i, swap[i] ? -crf_get(k1, i) : crf_get(k1, i));
        ok[i] = crf_get(h, i) >= 0x1p-60f && crf_get(h, i) <= 0x1p60f && crf_get(q0, i) >= 0x1p-20f &&
                crf_get(r, i) == crf_get(r2, i) && crf_get(z1, i) == crf_get(z2, i) && crf_get(s, i) == crf_get(sb, i) &&
                crf_get(c, i) == crf_get(cb, i) && crf_get(s2, i) == crf_get(s2b, i) && crf_get(k1, i) == crf_get(k2, i);
    }
    s2 = crf_add(s2, s2);
}
#endif  // LG_CRF_NO_QUICK
