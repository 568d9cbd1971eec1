"""The EPL lens's quick phases on the CPU: the polar frame (r, and the cosine
and sine of the rounded angle and of twice it, in one computation) and the
power with one exponent equal the double evaluations rounded once, bit for
bit, wherever the quick phase decides -- with the reciprocal estimates exact
and 2^-22 off either way, on points near and on the axes and diagonals, of
ordinary and extreme size (zeros, infinities and NaN quotients among them)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "native", "crf_polar.cpp")
RCP = {"exact": "(1.0f / (a))", "low": "((1.0f / (a)) * 0x1.fffffcp-1f)", "high": "((1.0f / (a)) * 0x1.000004p+0f)"}


@pytest.fixture(scope="module", params=sorted(RCP))
def polar(request, tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("crfp") / "crf_polar")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-DLG_CRF_HOST_RCP(a)=" + RCP[request.param],
                        SRC, "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


@pytest.mark.parametrize("size", [4, 28, 140])
def test_quick_phases(polar, size):
    out = subprocess.run([polar, "2000000", str(size), "7"], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr
    n, bad, und, pbad, prest = (int(v) for v in out.stdout.split())
    print(f"{und} of {n} frames and {prest} powers left to the one-value functions")
    assert bad == 0 and pbad == 0
