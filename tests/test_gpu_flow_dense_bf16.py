"""The training step's dense layers with BF16 activations, at widths on both
sides of each load's rule: weights in groups of 32 columns or not, layers that
start at multiples of 4, 8 and 16 bytes, activations in groups of four or not."""
import ctypes as C

import numpy as np
import pytest

import lensed_gb300 as lg
from oracle import flow_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,width", [(13, 128), (5, 32), (9, 36), (64, 64), (7, 31), (14, 96), (2, 64), (64, 33)])
def test_step_gradients_match_the_rounded_restatement(native, d, width):
    layers, hidden, n = 3, 2, 37
    rng = np.random.Generator(np.random.PCG64(d * 1000 + width))
    npar = lg.lib().lg_flow_nparams(d, layers, width, hidden)
    params = (rng.normal(size=npar) * 0.3 * np.sqrt(16 / width)).astype(np.float32)
    x = rng.normal(size=(n, d)).astype(np.float32)
    loss, grad = C.c_float(), np.zeros(npar, np.float32)
    fp = C.POINTER(C.c_float)
    assert lg.lib().lg_flow_loss_grad(0, d, layers, width, hidden, 1, params.ctypes.data_as(fp), x.ctypes.data_as(fp),
                                      n, C.byref(loss), grad.ctypes.data_as(fp)) == 0
    want_loss, want = flow_oracle.loss_grad(params.astype(np.float64), x.astype(np.float64), d, layers, width, hidden,
                                            act=flow_oracle.bf16)
    # FP32 sums as in the FP32 test (1e-4), and the few of up to 28416 activations
    # whose FP32 error (2^-22) crosses a rounding boundary (one in 2^13): 2^-8 in
    # one of 37 rows each, 4 of them 4e-4
    assert abs(loss.value - want_loss) <= 1e-3 * abs(want_loss)
    assert np.abs(grad - want).max() <= 1e-3 * np.abs(want).max()
