"""The programs of contexts for few candidates (split tiles and quadrature)
compose and compile without a GPU, for PSFs of one pixel to the widest that
is split and beyond."""
import numpy as np
import pytest

import lensed_gb300 as lg


@pytest.mark.parametrize("flags", [0, lg.LG_FLAG_FAST_MATH])
@pytest.mark.parametrize("pw,ph", [(1, 1), (12, 7), (49, 101), (50, 5)])
def test_small_contexts_compile(native, flags, pw, ph):
    lg.compile_check(96, 72, ["sie", "sersic", "sky"], psf=np.ones((ph, pw), np.float32), rule="sub3", flags=flags,
                     max_batch=1)
