"""Exact render with small blocks: those below 128 threads read the function
tables from global memory (an SM has room for only 7 copies in shared memory,
whatever the block), so their resident threads, and their time, are about
those of larger blocks: for 64 threads 1.1 times that of 256 (1.8 times with a
copy a block).  The values are the same."""
import numpy as np
import pytest

import lensed_gb300 as lg

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

OBJS = [("lens", "sie"), ("src", "sersic"), ("disk", "exponential"), ("sky", "sky")]


def test_small_blocks_keep_their_occupancy(native):
    n, B = 128, 512
    rng = np.random.Generator(np.random.PCG64(4))
    image = rng.normal(10, 3, (n, n)).astype(np.float32)
    ctx = lg.Context(image, np.full((n, n), 0.1, np.float32), OBJS, rule="sub3", max_batch=B)
    p = np.tile(np.array([64.0, 64, 25, 0.8, 30, 65, 63, 10, -3, 2, 0.7, 60, 65, 63, 12, -2.5, 0.7, 60, 10, 0, 0]), (B, 1))
    p[:, 2] *= np.linspace(0.9, 1.1, B)
    d = torch.from_numpy(ctx.to_map_order(p)).cuda()
    out = torch.empty(B, dtype=torch.float64, device="cuda")
    ms, logl = {}, {}
    for rt in (64, 128, 256):
        ctx.set_launch_shape(rt=rt)
        ms[rt] = min(ctx.profile(d.data_ptr(), B, out.data_ptr())[1] for _ in range(20))
        logl[rt] = out.cpu().numpy()
    print(ms)
    for rt in (64, 128):
        np.testing.assert_allclose(logl[rt], logl[256], rtol=1e-12, atol=0)  # grouping of the FP64 sums
        assert ms[rt] < 1.4 * ms[256], ms
    ctx.close()
