"""The set_params kernel's loops: models of more objects than a block has warps
(16) and too large for 32 candidates a block, the last block partly filled;
and a lens and a source that both carry image-plane priors, the source's being
deflected through that lens.  Each candidate's logL equals that of a call of
one candidate, whose object data come from the host one object after the
other."""
import numpy as np
import pytest

import lensed_gb300 as lg

pytestmark = pytest.mark.gpu


def check(objs, n, flags, B):
    rng = np.random.Generator(np.random.PCG64(B))
    image = rng.normal(10, 3, (n, n)).astype(np.float32)
    ctx = lg.Context(image, np.full((n, n), 0.1, np.float32), objs, rule="sub2", max_batch=B, flags=flags)
    assert ctx.host_set
    cube = rng.random((B, ctx.ndims))
    got, phys = ctx.eval_cube(cube)
    assert len(np.unique(got)) == B
    for b in range(B):
        one, p = ctx.eval_cube(cube[b])
        assert one[0] == got[b] and np.array_equal(p[0], phys[b])
    assert np.array_equal(ctx.eval_batch(phys), got)
    ctx.close()


@pytest.mark.parametrize("flags", [0, lg.LG_FLAG_STRICT_FP])
@pytest.mark.parametrize("sources,B", [(14, 33), (15, 32), (16, 70), (28, 70)])
def test_many_objects(native, flags, sources, B):
    objs = [("lens", "sie", ["24", "24", "unif 5 9", "unif 0.6 0.9", "unif 0 90"])]
    objs += [(f"s{i}", "gauss", [f"unif {18 + i % 5} {20 + i % 5}", f"unif {20 + i % 7} {21 + i % 7}", "unif 1 3",
                                 "unif -2 0", "unif 0.5 0.9", "unif 0 90"]) for i in range(sources)]
    check(objs + [("sky", "sky", ["unif 9 11", "0", "0"])], 40, flags, B)


@pytest.mark.parametrize("flags", [0, lg.LG_FLAG_FAST_MATH])
def test_image_plane_priors_of_lens_and_source(native, flags):
    objs = [("lens", "sie", ["image unif 20 28", "image unif 20 28", "unif 5 12", "unif 0.5 0.95", "unif 0 180"]),
            ("src", "sersic", ["image unif 10 20", "image unif 25 35", "unif 1 3", "unif -3 0", "unif 1 4",
                               "unif 0.5 1", "unif 0 180"])]
    check(objs, 48, flags, 40)
