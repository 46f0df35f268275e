"""GPU: an emission image is the same from run to run.

A block's warps take a packet's subtrees as they come free, so only the order in which FP64 subtree sums are added
may change; every FP32 rounding has to depend on the subtree alone.  An FP64 sum in another order is off by
about 2^-52 of itself and then rounded to FP32, so a value differs, by an ulp, with a chance of about
2^-52 / 2^-24 = 4e-9 a sum: none of the image's is expected to, and 3 values of 30,000 are allowed."""
import numpy as np
import pytest

import volprim_b200 as vp
from volprim_b200 import scenes
from volprim_b200.emission import render_emission

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w, h, spp", [(100, 100, 8), (280, 200, 1), (200, 250, 8)])  # blocks of 4, 4 and 2 warps
@pytest.mark.parametrize("precision", ["fast", "accurate"])
def test_runs_agree(vp_ctx, w, h, spp, precision):
    rng = np.random.default_rng(3)
    n = 12_000
    g = vp.Gaussians(rng.uniform(-0.6, 0.6, (n, 3)), np.exp(rng.normal(-2.5, 0.4, (n, 3))),
                     scenes.uniform_quaternions(rng, n), np.exp(rng.normal(0.0, 0.5, n)) * 2.0 / n)
    sc = vp.Scene(vp_ctx, g, 1.0)
    sc.set_emission(rng.uniform(0.0, 1.0, (n, 3)).astype(np.float32))
    env = vp.Environment(vp_ctx, constant=(0.7, 0.8, 0.9))
    cfg = vp.Config(num_samples_per_pixel=spp, image_width=w, image_height=h, seed=6, precision=precision)
    runs = [render_emission(sc, env, scenes.negz_camera(2.5, 40.0), cfg)[..., :3] for _ in range(4)]
    ref = runs[0]
    assert np.isfinite(ref).all() and ref.std() > 1e-3
    for r in runs[1:]:
        assert (r != ref).sum() <= 3e-4 * ref.size / 3 + 3, int((r != ref).sum())
        assert np.abs(r - ref).max() <= 2.0 ** -22 * np.abs(ref).max()
    env.close()
    sc.close()
