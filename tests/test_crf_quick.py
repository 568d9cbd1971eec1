"""The quick phases of the exact modules' exp, log, atan and atanh on the CPU:
dense windows where they switch path or table entry, with the reciprocal
estimate exact and two ulp off in either direction (the device's approximate
reciprocal lies between).  Every result must equal the double evaluation
rounded once, bit for bit: the quick phase may leave an input to the full
phase, never round it wrongly."""
import os
import struct
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "native", "crf_sweep.cpp")
RCP = {"exact": "(1.0f / (a))", "low": "((1.0f / (a)) * 0x1.fffffcp-1f)", "high": "((1.0f / (a)) * 0x1.000004p+0f)"}


def bits(x):
    return struct.unpack("I", struct.pack("f", x))[0]


@pytest.fixture(scope="module", params=sorted(RCP))
def sweep(request, tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("crfq") / "crf_sweep")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fopenmp",
                        "-DLG_CRF_HOST_RCP(a)=" + RCP[request.param], SRC, "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(fn, start, stop, step=1):
        out = subprocess.run([exe, str(fn), str(start), str(stop), str(step)], capture_output=True, text=True,
                             timeout=600)
        assert out.returncode == 0, out.stderr
        n, bad, nin, slow = (int(v) for v in out.stdout.split())
        return n, bad, out.stderr

    return run


WINDOWS = [
    (0, bits(86.9), bits(87.1)), (0, bits(-86.9), bits(-87.1)),    # exp: the ends of the quick range
    (0, bits(1e-4), bits(7e-4)), (0, bits(-1e-4), bits(-7e-4)),    # exp: results next to 1, k = 0 and 1
    (0, bits(0.692), bits(0.694)),                                 # exp: results next to 2
    (0, 0, 2000000), (0, bits(-0.0), bits(-0.0) + 2000000),        # exp: zero and subnormals
    (1, bits(0.999), bits(1.001)),                                 # log near 1: left to the full phase
    (1, bits(1.999), bits(2.001)), (1, bits(0.4995), bits(0.5005)),  # log: the ends of the mantissa's range
    (1, bits(2.0 ** -126) - 1000000, bits(2.0 ** -126) + 1000000),  # log: the smallest normal
    (1, bits(3.4e38), bits(float("inf")) + 1000),                  # log: the largest, infinite, NaN
    (2, bits(0.999), bits(1.001)), (2, bits(9e-4), bits(3e-3)),    # atan: both sides of 1; the first entries
    (2, bits(1.999), bits(2.001)),                                 # atan: the end of the table
    (1, bits(2.0 ** 91) - 100000, bits(2.0 ** 91) + 100000),       # log: the ends of the quick range
    (1, bits(2.0 ** -90) - 100000, bits(2.0 ** -90) + 100000),
    (2, bits(8e37), bits(float("inf")) + 1000),                    # atan: 1/a flushed to 0, infinite, NaN
    (3, bits(0.899), bits(0.901)), (3, bits(9e-4), bits(3e-3)),    # atanh: the end of the quick range; first entries
    (3, bits(0.999), bits(1.001)),                                 # atanh: 1 and above
]


@pytest.mark.parametrize("fn,lo,hi", WINDOWS)
def test_windows(sweep, fn, lo, hi):
    lo, hi = min(lo, hi), max(lo, hi)
    n, bad, err = sweep(fn, lo, hi, 1 + (hi - lo) // 1000000)
    assert n > 10000 and bad == 0, err


@pytest.mark.parametrize("fn", [0, 1, 2, 3])
def test_stride(sweep, fn):
    n, bad, err = sweep(fn, 0, 1 << 32, 1009)
    assert bad == 0, err
