"""The EPL lens's quick phases decide nearly all ordinary points and powers, so
that the comparisons of what they decide mean something.  Of the harness's
points of ordinary size one in eight each has an axis angle of 2^-24 to 1 (below
2^-20, or about 2^-14 where an absolute margin is left of the result, all are
undecided: 2, 2 and 5% of all points) and one in 64 is on a diagonal (cos 2phi
of nearly 0: undecided): 11%; of the powers 2 (1.5 2^-32 |y|) / 2^-23 for the mean
|y| of 1.5: 1%."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "native", "crf_polar.cpp")


def test_undecided_fractions(tmp_path):
    exe = str(tmp_path / "crf_polar")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", SRC, "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe, "1000000", "4", "3"], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr
    n, bad, und, pbad, prest = (int(v) for v in out.stdout.split())
    assert bad == 0 and pbad == 0
    assert und < 0.15 * n and prest < 0.02 * n
