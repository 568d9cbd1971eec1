// Route the float elementary functions of the following plugin code to the
// correctly rounded versions of the prelude.
#define expf(x) lg_cr_expf(x)
#define exp2f(x) lg_cr_exp2f(x)
#define expm1f(x) lg_cr_expm1f(x)
#define logf(x) lg_cr_logf(x)
#define log2f(x) lg_cr_log2f(x)
#define log10f(x) lg_cr_log10f(x)
#define log1pf(x) lg_cr_log1pf(x)
#define powf(x, y) lg_cr_powf(x, y)
#define sinf(x) lg_cr_sinf(x)
#define cosf(x) lg_cr_cosf(x)
#define tanf(x) lg_cr_tanf(x)
#define sincosf(x, s, c) lg_cr_sincosf(x, s, c)
#define asinf(x) lg_cr_asinf(x)
#define acosf(x) lg_cr_acosf(x)
#define atanf(x) lg_cr_atanf(x)
#define atan2f(y, x) lg_cr_atan2f(y, x)
#define sinhf(x) lg_cr_sinhf(x)
#define coshf(x) lg_cr_coshf(x)
#define tanhf(x) lg_cr_tanhf(x)
#define asinhf(x) lg_cr_asinhf(x)
#define acoshf(x) lg_cr_acoshf(x)
#define atanhf(x) lg_cr_atanhf(x)
#define tgammaf(x) lg_cr_tgammaf(x)
#define lgammaf(x) lg_cr_lgammaf(x)
#define cbrtf(x) lg_cr_cbrtf(x)
#define erff(x) lg_cr_erff(x)
#define erfcf(x) lg_cr_erfcf(x)

#ifdef LG_CRF_NO_QUICK
// The set_params module: the functions that lg_crfloat.cuh evaluates in
// single-precision arithmetic give the same values (the double evaluation
// rounded once) without GB300's slow FP64 -- one candidate's Sersic object
// took 8 us in it, most of it in four logarithms, a sine and a cosine.
LG_DEV float lg_set_sinf(float x)
{
    float s, c;
    lg_crf_sincos(x, &s, &c);
    return s;
}
LG_DEV float lg_set_cosf(float x)
{
    float s, c;
    lg_crf_sincos(x, &s, &c);
    return c;
}
#undef expf
#undef logf
#undef powf
#undef sinf
#undef cosf
#undef sincosf
#undef atanf
#undef atan2f
#undef atanhf
#define expf(x) crf_full_exp(x)
#define logf(x) crf_full_log(x)
#define powf(x, y) lg_crf_pow(x, y)
#define sinf(x) lg_set_sinf(x)
#define cosf(x) lg_set_cosf(x)
#define sincosf(x, s, c) lg_crf_sincos(x, s, c)
#define atanf(x) crf_full_atan(x)
#define atan2f(y, x) lg_crf_atan2(y, x)
#define atanhf(x) crf_full_atanh(x)
#endif
