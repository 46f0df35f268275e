"""GPU: which form takes a wavefront image's paths -- threads over the 8-wide BVH, a warp on each over the BVH32, the
launch that ends a batch -- goes by how many are left and by what the scene holds.  Every route against the warp
engine, at both sides of its lines; the tolerance is test_gpu_trace8.py's (the same chords, FP64 sums rounded once:
1e-5 of the image's mean)."""
import numpy as np
import pytest

import test_gpu_trace8 as T
import volprim_b200 as vp
from volprim_b200 import scenes

pytestmark = pytest.mark.gpu


def compare(ctx, g, w, h, bounces, sigma=1.0, camera=None, **kw):
    sc = vp.Scene(ctx, g, sigma)
    env = vp.Environment(ctx, rgb=scenes.procedural_env(64, 32, sun_radiance=50.0, sun_radius_deg=8.0))
    out = {}
    for engine in ("wavefront", "warp"):
        cfg = vp.Config(num_samples_per_pixel=1, image_width=w, image_height=h, seed=5, engine=engine,
                        max_bounces=bounces, rr_depth=4, **kw)
        out[engine] = vp.Renderer(cfg, sc, camera or scenes.negz_camera(3.0, 40.0), env=env, ctx=ctx).render()[..., :3]
    info = sc.info()
    env.close()
    sc.close()
    T.check(out["wavefront"], out["warp"])
    return info


# extend by threads above 65,536 paths, shadow above 16,384; the last 2,368 or (above 32 bounces) 4,736 in one launch
@pytest.mark.parametrize("w, h", [(257, 256), (256, 256), (145, 113), (128, 128), (74, 64), (74, 65), (37, 64), (37, 65)])
@pytest.mark.parametrize("bounces", [16, 40])
def test_differing_albedos(vp_ctx, w, h, bounces):
    compare(vp_ctx, T.gaussians(500, 7), w, h, bounces, sigma=2.0, hg_g=0.3, camera=scenes.negz_camera(1.2, 30.0))


@pytest.mark.parametrize("w, h", [(74, 65), (37, 65), (37, 64)])
@pytest.mark.parametrize("mixed", [False, True])
def test_too_deep_for_the_8_wide_tree(vp_ctx, w, h, mixed):
    compare(vp_ctx, T.gaussians(600, 3, "nested", mixed), w, h, 16, hg_g=0.0)
