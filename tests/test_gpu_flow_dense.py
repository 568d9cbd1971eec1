"""The training step's dense layers at the widths where their loads change:
weights in groups of 32 columns or not, layers that start at multiples of 4,
8 and 16 bytes, activations in groups of four or not."""
import ctypes as C

import numpy as np
import pytest

import lensed_gb300 as lg
from oracle import flow_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,width", [(13, 128), (5, 32), (9, 36), (64, 64), (7, 31), (14, 96), (2, 64), (64, 33)])
def test_step_gradients_match_the_restatement(native, d, width):
    layers, hidden, n = 3, 2, 37
    rng = np.random.Generator(np.random.PCG64(d * 1000 + width))
    npar = lg.lib().lg_flow_nparams(d, layers, width, hidden)
    params = (rng.normal(size=npar) * 0.3 * np.sqrt(16 / width)).astype(np.float32)
    x = rng.normal(size=(n, d)).astype(np.float32)
    loss, grad = C.c_float(), np.zeros(npar, np.float32)
    fp = C.POINTER(C.c_float)
    assert lg.lib().lg_flow_loss_grad(0, d, layers, width, hidden, 0, params.ctypes.data_as(fp), x.ctypes.data_as(fp),
                                      n, C.byref(loss), grad.ctypes.data_as(fp)) == 0
    want_loss, want = flow_oracle.loss_grad(params.astype(np.float64), x.astype(np.float64), d, layers, width, hidden)
    # FP32 sums of up to 128 terms through 9 dense layers and back: 128 x 9 x 2^-24
    assert abs(loss.value - want_loss) <= 1e-4 * abs(want_loss)
    assert np.abs(grad - want).max() <= 1e-4 * np.abs(want).max()
