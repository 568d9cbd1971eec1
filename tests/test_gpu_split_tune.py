"""The tuner and split tiles (contexts of few convolution tiles): which
contexts use them, that LG_FLAG_AUTOTUNE keeps or times them, and that the
file of tuned shapes carries the choice (a line without it has whole tiles)."""
import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest

import lensed_gb300 as lg

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
P = np.array([48.0, 36, 14, 0.8, 30, 50, 37, 4, -3, 2, 0.7, 60, 10, 0, 0])


def context(B, flags=0, priors=True, w=96, h=72, psf=(11, 11)):
    rng = np.random.Generator(np.random.PCG64(w + h))
    image = rng.normal(10, 3, (h, w)).astype(np.float32)
    val = [(f"unif {v - 0.05} {v + 0.05}" if v else "0") if priors else None for v in P]
    objs = [("lens", "sie", val[:5]), ("src", "sersic", val[5:12]), ("sky", "sky", val[12:])]
    if not priors:
        objs = [(i, p, None) for i, p, _ in objs]
    return lg.Context(image, np.full((h, w), 0.1, np.float32), objs, psf=rng.uniform(0.1, 1, psf).astype(np.float32),
                      rule="sub3", max_batch=B, flags=flags)


def logl(ctx):
    return ctx.eval_batch(ctx.to_map_order(P[None]))[0]


@pytest.mark.parametrize("w,h,pw,ph", [(64, 128, 25, 25), (33, 65, 3, 2), (31, 7, 12, 12), (101, 77, 1, 1),
                                       (96, 63, 49, 17), (40, 200, 8, 31), (256, 256, 25, 25)])
def test_contexts_that_split(native, w, h, pw, ph):
    for B, flags, split in ((1, 0, True), (2, lg.LG_FLAG_FAST_MATH, True), (1, lg.LG_FLAG_STRICT_FP, False), (1024, 0, False)):
        ctx = context(B, flags, w=w, h=h, psf=(ph, pw))
        assert ctx.split_tiles == split
        ctx.close()


def test_untuned_context_keeps_the_default(native):
    plain, tuned = context(1), context(1, lg.LG_FLAG_AUTOTUNE, priors=False)
    assert tuned.tune_report.startswith("not tuned")
    assert tuned.split_tiles and tuned.launch_shape == plain.launch_shape
    assert logl(tuned) == logl(plain)


def test_split_tiles_are_timed_and_kept_in_the_file(native, tmp_path):
    cache = tmp_path / "tune.txt"
    script = textwrap.dedent(f"""
        import sys
        sys.path.insert(0, {ROOT!r})
        sys.path.insert(0, {os.path.join(ROOT, 'tests')!r})
        import lensed_gb300 as lg
        from test_gpu_split_tune import context, logl
        ctx, ref = context(1, lg.LG_FLAG_AUTOTUNE), context(1)
        assert abs(logl(ctx) / logl(ref) - 1) < 1e-12
        rep = ctx.tune_report
        print(rep.split()[0], ", split" in rep.splitlines()[0], ", split: render" in rep, ctx.split_tiles)
    """)

    def run():
        r = subprocess.run([sys.executable, "-c", script], env=dict(os.environ, LG_TUNE_CACHE=str(cache)),
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr
        return r.stdout.split()

    first = run()
    assert first[0] == "tuned" and first[2] == "True" and first[1] == first[3]
    key = cache.read_text().split()[0]
    for line, split in ((f"{key} 256 2 4 32 64 8 1 1\n", "True"), (f"{key} 256 2 4 32 64 8 1\n", "False"),
                        (f"{key} 256 2 4 32 16 4 0\n", "False")):
        cache.write_text(line)
        assert run() == ["cached", split, "False", split]
