"""GPU: a render of max_bounces = 0 traces no vertex, so its image is black in every engine, with and without
adaptive sampling (whose batches queue their paths on a route of their own)."""
import numpy as np
import pytest

import volprim_b200 as vp
from volprim_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", ["wavefront", "warp", "megakernel"])
@pytest.mark.parametrize("albedo", [0.0, 0.8])
@pytest.mark.parametrize("threshold", [0.0, 1e-3])
def test_no_bounces_no_light(vp_ctx, engine, albedo, threshold):
    g = scenes.absorption_gaussians(200, 1)
    g.albedo = np.full((200, 3), albedo, np.float32)
    sc = vp.Scene(vp_ctx, g, 1.0)
    env = vp.Environment(vp_ctx, constant=(1.0, 1.0, 1.0))
    cfg = vp.Config(num_samples_per_pixel=4, image_width=37, image_height=29, seed=2, max_bounces=0, engine=engine,
                    adaptive_threshold=threshold, adaptive_min_samples=64, batch_spp=2)
    img = vp.ProgressiveImage(vp_ctx, 37, 29)
    st = img.accumulate(sc, env, scenes.negz_camera(3.0, 40.0), cfg, 0, 4)
    assert st["paths"] == 37 * 29 * 4 and st["device_status"] == 0
    assert np.all(img.read()[..., :3] == 0.0)
    assert np.all(img.read_welford(m2=False)[1] == 4)
    img.close()
    env.close()
    sc.close()
