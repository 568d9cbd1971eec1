"""The quick phases of the correctly rounded functions on the CPU with their
packed products (crf_mulx) fused into the sums that take them, in every
combination, as the device's assembler may fuse them: exp, log, atan, atanh,
the EPL lens's power and polar frame equal the double evaluations rounded
once, bit for bit."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "native", "crf_contract.cpp")


def test_contracted_products(tmp_path):
    exe = str(tmp_path / "crf_contract")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", SRC, "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe, "200000", "5"], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr
    sums, bad = zip(*(map(int, line.split()) for line in out.stdout.splitlines()))
    assert len(bad) == 6 and sums[2] > 0 and sums[5] > 0  # (atan and the frame do add such products)
    assert bad == (0,) * 6
