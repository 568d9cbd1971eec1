"""Generate lg_crf_tables.cuh, the tables, and lg_crf_consts.cuh, their
offsets and the split constants, of the correctly rounded single-precision
functions in lg_crfloat.cuh.

Every value is computed with mpmath at 60 significant digits and rounded to
float (round to nearest even) once; a "double-word" pair (hi, lo) holds
hi = RN(v) and lo = RN(v - hi).  All tables are one array of 64-bit words, two
floats each; the library holds it on the device and NVRTC modules reach it
through a pointer, so that no model's compilation has to read them.

  exp   T_j = 2^(j/64), j = 0..63, as (hi, lo)                (Tang 1989);
        for the quick phase 2^((j + 1)/1024), j = 0..1023, as (hi, lo + D)
        with D the half-width of its rounding interval
  log   for the 1024 intervals of the mantissa m in [0.75, 1.5) (512 of
        width 2^-11 below 1, 512 of width 2^-10 above): c_j = RN(1 / centre)
        (c = 1 for the two intervals next to 1) and -ln(c_j) as (hi, lo)
        (Tang 1990); for the quick phase ln(2)/2 - ln(c) of every c of 11
        significant bits from 1/2 - 2^-12 to 1, as (hi, lo + D) with hi a
        multiple of 2^-18
  atan  atan(j/512), j = 0..1024, as (hi, lo)
  atanh atanh(j/512), j = 0..461, as (hi, lo), padded to 512 entries
  sin/cos  sin(j/256) and cos(j/256), j = -201..201, as (hi, lo) pairs

Run:  python lensed_gb300/device/make_crf_tables.py
"""
import os
import struct

import mpmath as mp

mp.mp.dps = 60
HERE = os.path.dirname(os.path.abspath(__file__))


def rn(v) -> float:
    """Round an mpmath value to the nearest float32 (ties to even)."""
    d = float(v)  # nearest double; re-round with the exact remainder
    f = struct.unpack("f", struct.pack("f", d))[0]
    # struct rounds the double to float with ties-to-even; correct a double
    # rounding by comparing against the exact value
    if f != 0 and mp.isfinite(v):
        lo_n = struct.unpack("f", struct.pack("I", struct.unpack("I", struct.pack("f", f))[0] - 1))[0]
        hi_n = struct.unpack("f", struct.pack("I", struct.unpack("I", struct.pack("f", f))[0] + 1))[0]
        best = min((abs(mp.mpf(c) - v), c) for c in (lo_n, f, hi_n))
        f = best[1]
    return f


def split(v):
    hi = rn(v)
    lo = rn(v - mp.mpf(hi))
    return hi, lo


def lit(f: float) -> str:
    if f == 0:
        return "0.0f"
    h = float.hex(f)  # e.g. 0x1.5d58980000000p-1
    mant, exp = h.split("p")
    if "." in mant:
        mant = mant.rstrip("0").rstrip(".")
    return f"{mant}p{exp}f"


def word(*fs) -> str:
    """Two (four) floats as one (two) 64-bit words, the first in the low half."""
    b = [struct.unpack("I", struct.pack("f", f))[0] for f in fs]
    return ", ".join(f"0x{b[i + 1]:08x}{b[i]:08x}u" for i in range(0, len(b), 2))


def main():
    head = "// generated by lensed_gb300/device/make_crf_tables.py -- do not edit"
    tabs = {}
    # exp: 2^(j/64)
    rows = []
    for j in range(64):
        hi, lo = split(mp.power(2, mp.mpf(j) / 64))
        rows.append(word(hi, lo))
    tabs["EXP"] = rows
    # log: (c, -ln c hi, -ln c lo, 0)
    rows = []
    for j in range(1024):
        if j < 512:
            m0, w = mp.mpf(0.75) + j * mp.mpf(2) ** -11, mp.mpf(2) ** -11
        else:
            m0, w = 1 + (j - 512) * mp.mpf(2) ** -10, mp.mpf(2) ** -10
        c = 1.0 if j in (511, 512) else rn(1 / (m0 + w / 2))
        hi, lo = split(-mp.log(mp.mpf(c)))
        rows.append(word(c, hi, lo, 0.0))
    tabs["LOG"] = rows
    # exp, quick phase: 2^((j + 1)/1024) as (hi, lo + D)
    D = mp.mpf(float.fromhex("0x1.ap-35"))
    rows = []
    for j in range(1024):
        v = mp.power(2, mp.mpf(j + 1) / 1024)
        hi = rn(v)
        rows.append(word(hi, rn(v - mp.mpf(hi) + D)))
    quick = {"EXP": rows}
    # log, quick phase: ln2/2 - ln(c), c = float with bit pattern 0x3effe000 + j
    # 2^13, as (hi, lo + D)
    D = mp.mpf(float.fromhex("0x1.6p-34"))
    rows = []
    for j in range(1026):
        c = struct.unpack("f", struct.pack("I", 0x3EFFE000 + (j << 13)))[0]
        v = mp.log(2) / 2 - mp.log(mp.mpf(c))
        hi = mp.floor(v * 2 ** 18 + mp.mpf(0.5)) / 2 ** 18
        assert mp.mpf(rn(hi)) == hi
        rows.append(word(rn(hi), rn(v - hi + D)))
    quick["LOG"] = rows
    # atan(j/512)
    rows = []
    for j in range(1025):
        hi, lo = split(mp.atan(mp.mpf(j) / 512))
        rows.append(word(hi, lo))
    quick["ATAN"] = rows
    # atanh(j/512), j = 0..461, as (hi, lo), padded to 512 entries
    rows = []
    for j in range(462):
        hi, lo = split(mp.atanh(mp.mpf(j) / 512))
        rows.append(word(hi, lo))
    rows += [word(0.0, 0.0)] * 50
    quick["ATANH"] = rows
    # sin / cos(j/256), j = -201..201, as (sin hi, sin lo, cos hi, cos lo)
    rows = []
    for j in range(-201, 202):
        a = mp.mpf(j) / 256
        sh, sl = split(mp.sin(a))
        ch, cl = split(mp.cos(a))
        rows.append(word(sh, sl, ch, cl))
    tabs["SC"] = rows
    # first word of each table; those of the quick phases side by side, as
    # they are copied to shared memory (LG_CRF_Q_*: relative to LG_CRF_AT_Q)
    words, defs, q = [], [], 0
    for name in ("EXP", "LOG", "SC"):
        defs.append(f"#define LG_CRF_AT_{name} {len(words)}")
        words += [w.strip() for r in tabs[name] for w in r.split(",")]
        words += [word(0.0, 0.0)] * (len(words) % 2)
    defs.append(f"#define LG_CRF_AT_Q {len(words)}")
    for name in ("EXP", "LOG", "ATAN", "ATANH"):
        defs.append(f"#define LG_CRF_Q_{name} {q}")
        words += quick[name]
        q += len(quick[name])
    words += [word(0.0, 0.0)] * (q % 2)
    defs.append(f"#define LG_CRF_Q_ENTRIES {q + q % 2}")
    # split constants
    consts = {}
    l64 = mp.log(2) / 64
    consts["LG_CRF_EXP_INVL"] = rn(64 / mp.log(2))
    consts["LG_CRF_EXP_LHI"], consts["LG_CRF_EXP_LLO"] = split(l64)
    # quick phases: ln2/1024 = L_hi + L_lo; ln2 2^-23 = (multiple of 2^-40) + rest
    consts["LG_CRF_QEXP_INVL"] = rn(1024 / mp.log(2))
    consts["LG_CRF_QEXP_LHI"], consts["LG_CRF_QEXP_LLO"] = split(mp.log(2) / 1024)
    h = mp.floor(mp.log(2) * 2 ** 17 + mp.mpf(0.5)) / 2 ** 17
    consts["LG_CRF_QLN2_HI"], consts["LG_CRF_QLN2_LO"] = rn(h * mp.mpf(2) ** -23), rn((mp.log(2) - h) * mp.mpf(2) ** -23)
    consts["LG_CRF_LN2_HI"], consts["LG_CRF_LN2_LO"] = split(mp.log(2))
    consts["LG_CRF_PIO2_HI"], consts["LG_CRF_PIO2_LO"] = split(mp.pi / 2)
    # sin / cos argument reduction: 2/pi, and pi/2 = P1 + P2 + P3 with P1
    # and P2 of 17 significant bits (k P1, k P2 exact for |k| < 2^7)
    consts["LG_CRF_INV_PIO2"] = rn(2 / mp.pi)
    p1 = mp.floor(mp.pi / 2 * 2 ** 16 + mp.mpf(0.5)) / 2 ** 16
    p2 = mp.floor((mp.pi / 2 - p1) * 2 ** 33 + mp.mpf(0.5)) / 2 ** 33
    consts["LG_CRF_PIO2_1"], consts["LG_CRF_PIO2_2"] = rn(p1), rn(p2)
    assert mp.mpf(rn(p1)) == p1 and mp.mpf(rn(p2)) == p2
    consts["LG_CRF_PIO2_3"] = rn(mp.pi / 2 - p1 - p2)
    # exp(x) rounds to 0 for x <= LG_CRF_EXP_ZERO (e^x <= 2^-150, the tie at
    # 2^-150 going to the even value 0): the largest such float
    t = mp.log(mp.mpf(2) ** -150)
    f = rn(t)
    if mp.mpf(f) > t:  # e^f > 2^-150: step one float down (away from zero)
        f = struct.unpack("f", struct.pack("I", struct.unpack("I", struct.pack("f", f))[0] + 1))[0]
    consts["LG_CRF_EXP_ZERO"] = f
    defs += [f"#define {k} ({lit(v)})" for k, v in consts.items()]
    for name, lines in (("consts", ["// Table offsets and split constants of the correctly rounded functions."] + defs),
                        ("tables", ["// Tables of the correctly rounded functions (lg_crfloat.cuh).",
                                    f"LG_CRF_TABLE(lg_crf_words, {len(words)}) = {{\n    " + ",\n    ".join(words) + "};"])):
        with open(os.path.join(HERE, f"lg_crf_{name}.cuh"), "w") as fh:
            fh.write("\n".join([head] + lines) + "\n")


if __name__ == "__main__":
    main()
