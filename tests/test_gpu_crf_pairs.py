"""The EPL lens's quick phases on the GPU as the render runs them, on pairs:
the polar frame (r, cos and sin of the rounded angle and of twice it) wherever
it decides, and the power with one exponent, equal the double evaluations
rounded once, bit for bit, on 2^28 pairs each -- axes, diagonals, quotients
next to 2^-20 and H next to 2^-60 and 2^60 among the points."""
import ctypes as C

import pytest

import lensed_gb300 as lg

pytestmark = pytest.mark.gpu


def sweep(fn, n):
    bad, first = C.c_ulonglong(), (C.c_uint * 8)()
    assert lg.lib().lg_probe_crf_sweep(0, fn, C.c_ulonglong(0), C.c_ulonglong(n), C.byref(bad), first, 8) == 0
    return bad.value, [first[i] for i in range(min(bad.value, 8))]


@pytest.mark.parametrize("fn", [9, 10])
def test_pairs_equal_the_double_evaluation(native, fn):
    bad, first = sweep(fn, 1 << 28)
    assert bad == 0, first

