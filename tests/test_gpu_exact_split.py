"""The exact mode's quadrature split with its values gathered a few points at
a time, and its function tables in shared memory or (where the gathered
values leave no room) in global memory: images and logL equal the unsplit
default shape's bit for bit, for rules around the chunk sizes, one or several
candidates a block, with and without a PSF."""
import numpy as np
import pytest

import lensed_gb300 as lg
from lensed_gb300 import workloads

pytestmark = pytest.mark.gpu

OBJS = [("lens", "epl_plus_shear"), ("src", "sersic"), ("sky", "sky")]
TRUTH = [31.0, 22.0, 9.0, 1.1, 0.8, 40.0, 0.02, -0.01, 32.0, 21.0, 3.0, -3.0, 2.0, 0.7, 60.0, 10.0, 0.01, -0.02]
# (render threads, pixels a group, split): chunk of one, of several, of all points; tables global in the last
SHAPES = [(32, 2, 8), (128, 2, 2), (128, 4, 4), (512, 2, 2), (1024, 2, 4), (1024, 6, 2)]


def params(B):
    p = np.tile(np.array(TRUTH), (B, 1))
    p[:, 2] += np.linspace(-0.5, 0.5, B)
    p[:, 9] += np.linspace(0.4, -0.4, B)
    return p


@pytest.mark.parametrize("rule", ["point", "sub3", "g3k7"])
@pytest.mark.parametrize("psf", [0, 9])
def test_split_shapes_equal_default(native, rule, psf):
    rng = np.random.Generator(np.random.PCG64(5))
    image = rng.normal(10, 3, (45, 63)).astype(np.float32)
    weight = np.full_like(image, 0.1)
    ctx = lg.Context(image, weight, OBJS, psf=workloads.psf_gauss_wings(psf, 2.0) if psf else None, rule=rule,
                     max_batch=40)
    ctx.set_launch_shape(rt=128, rppt=2, qs=1)
    p = ctx.to_map_order(params(40))
    want, images = ctx.eval_batch(p), ctx.render(p[7])
    for rt, rppt, qs in SHAPES:
        ctx.set_launch_shape(rt=rt, rppt=rppt, qs=qs)
        got = ctx.eval_batch(p)
        assert np.allclose(got, want, rtol=1e-13, atol=0), (rt, rppt, qs)  # (order of the FP64 sum)
        if psf:  # the convolution's tiles are the same: no other order
            assert np.array_equal(got, want), (rt, rppt, qs)
        for a, b in zip(ctx.render(p[7]), images):
            assert np.array_equal(a, b), (rt, rppt, qs)
    ctx.close()
