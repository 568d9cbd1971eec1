"""Contexts for one or a few candidates split their convolution tiles over
clusters of blocks (and, in the exact mode, the quadrature over threads): logL
and the dumped images equal those of the whole-tile shape bit for bit, for
images smaller than a tile, with ragged edges in either direction, odd, even
and wide PSFs, in the exact and the fast mode."""
import numpy as np
import pytest

import lensed_gb300 as lg
from lensed_gb300 import workloads

pytestmark = pytest.mark.gpu

OBJS = [("lens", "sie"), ("src", "sersic"), ("sky", "sky")]


def params(w, h, B):
    p = np.tile(np.array([w / 2, h / 2, min(w, h) / 5 + 1, 0.8, 30.0, w / 2 + 1, h / 2 - 1, min(w, h) / 12 + 1, -3.0, 2.0, 0.7,
                          60.0, 10.0, 0.01, -0.02]), (B, 1))
    p[:, 2] *= np.linspace(0.9, 1.1, B)
    return p


@pytest.mark.parametrize("flags", [0, lg.LG_FLAG_FAST_MATH])
@pytest.mark.parametrize("w,h,pw,ph", [(64, 128, 25, 25), (33, 65, 3, 2), (31, 7, 12, 12), (101, 77, 1, 1), (96, 63, 49, 17),
                                       (40, 200, 8, 31), (256, 256, 25, 25)])
def test_split_equals_whole_tiles(native, flags, w, h, pw, ph):
    rng = np.random.Generator(np.random.PCG64(w * h))
    image = rng.normal(10, 3, (h, w)).astype(np.float32)
    weight = rng.uniform(0, 0.2, (h, w)).astype(np.float32)
    weight[rng.random((h, w)) < 0.1] = 0
    psf = rng.uniform(0.1, 1, (ph, pw)).astype(np.float32)
    for B in (1, 2):
        ctx = lg.Context(image, weight, OBJS, psf=psf, rule="sub3", max_batch=B, flags=flags)
        p = ctx.to_map_order(params(w, h, B))
        got, images = ctx.eval_batch(p), ctx.render(p[-1])
        assert np.array_equal(ctx.eval_batch(p), got)  # the counters are back to zero
        shape = dict(ctx.launch_shape, qs=1)
        ctx.set_launch_shape(**shape)  # a given shape has whole tiles
        assert np.array_equal(ctx.eval_batch(p), got)
        for a, b in zip(ctx.render(p[-1]), images):
            assert np.array_equal(a, b)
        ctx.close()
