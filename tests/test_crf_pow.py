"""The exact modules' paired power (lg_crf_pow1) on the CPU where its error is
largest: equal to the double evaluation rounded once, bit for bit.  The first
power is one whose rounding an interval of 2^-32 |y| decides wrongly when the
logarithm's r and t are summed to a float before y times it is taken."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "native", "crf_pow.cpp")


def test_largest_errors(tmp_path):
    exe = str(tmp_path / "crf_pow")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", SRC, "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe, "20000000", "2", "0x1.f2e4bcp-88", "-0x1.14750ep+0"], capture_output=True, text=True,
                         timeout=600)
    assert out.returncode == 0, out.stderr
    n, bad = map(int, out.stdout.split())
    assert n > 100000
    assert bad == 0, out.stderr
