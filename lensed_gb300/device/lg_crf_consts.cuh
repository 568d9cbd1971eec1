// generated by lensed_gb300/device/make_crf_tables.py -- do not edit
// Table offsets and split constants of the correctly rounded functions.
#define LG_CRF_AT_EXP 0
#define LG_CRF_AT_LOG 64
#define LG_CRF_AT_SC 2112
#define LG_CRF_AT_Q 2918
#define LG_CRF_Q_EXP 0
#define LG_CRF_Q_LOG 1024
#define LG_CRF_Q_ATAN 2050
#define LG_CRF_Q_ATANH 3075
#define LG_CRF_Q_ENTRIES 3588
#define LG_CRF_EXP_INVL (0x1.715476p+6f)
#define LG_CRF_EXP_LHI (0x1.62e43p-7f)
#define LG_CRF_EXP_LLO (-0x1.05c61p-35f)
#define LG_CRF_QEXP_INVL (0x1.715476p+10f)
#define LG_CRF_QEXP_LHI (0x1.62e43p-11f)
#define LG_CRF_QEXP_LLO (-0x1.05c61p-39f)
#define LG_CRF_QLN2_HI (0x1.62e4p-24f)
#define LG_CRF_QLN2_LO (0x1.7f7d1cp-43f)
#define LG_CRF_LN2_HI (0x1.62e43p-1f)
#define LG_CRF_LN2_LO (-0x1.05c61p-29f)
#define LG_CRF_PIO2_HI (0x1.921fb6p+0f)
#define LG_CRF_PIO2_LO (-0x1.777a5cp-25f)
#define LG_CRF_INV_PIO2 (0x1.45f306p-1f)
#define LG_CRF_PIO2_1 (0x1.922p+0f)
#define LG_CRF_PIO2_2 (-0x1.2aeep-18f)
#define LG_CRF_PIO2_3 (-0x1.e973dcp-35f)
#define LG_CRF_EXP_ZERO (-0x1.9fe36ap+6f)
