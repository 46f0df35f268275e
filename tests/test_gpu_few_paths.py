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


def has_8_wide_tree(info):
    n = info["count"]
    return info["device_bytes"] > 132 * n + 1024 * info["wide_nodes"] + 64 * max(n - 1, 1)


def box(n, seed, size, mixed):
    rng = np.random.default_rng(seed)
    scale = np.exp(rng.normal(np.log(size), 0.4, (n, 3)))
    dens = np.exp(rng.normal(0.0, 0.5, n)) * 200.0 * size * size / n
    albedo = rng.uniform(0.2, 0.95, (n, 3)) if mixed else np.full((n, 3), 0.8)
    return vp.Gaussians(*(a.astype(np.float32) for a in (rng.uniform(-1, 1, (n, 3)), scale,
                                                         scenes.uniform_quaternions(rng, n), dens, albedo)))


# Gaussians that fill 0.06, 0.11, 0.16, 0.25 and 0.4 of a box of side 2: above 0.1 the tail takes fewer paths (ACCURATE:
# 0.02), above 0.2 there is no 8-wide tree, unless one node holds all (8 Gaussians)
@pytest.mark.parametrize("n, size, tree", [(300, 0.1, True), (300, 0.15, True), (300, 0.2, True), (300, 0.3, False),
                                           (33, 0.5, False), (9, 0.5, False), (8, 0.5, True), (1, 0.5, True)])
@pytest.mark.parametrize("precision", ["fast", "accurate"])
@pytest.mark.parametrize("mixed", [False, True])
def test_gaussians_as_large_as_the_scene(vp_ctx, n, size, tree, precision, mixed):
    info = compare(vp_ctx, box(n, 11, size, mixed), 150, 130, 40 if mixed else 12, precision=precision, hg_g=0.0)
    assert has_8_wide_tree(info) == tree


@pytest.mark.parametrize("far", [0.0, 1e4])
def test_many_identical_boxes(vp_ctx, far):
    """Small Gaussians, twenty in each of 60 places: a tree of equal boxes, near the origin and far from it (the
    share of the scene they fill does not change with its place)."""
    rng = np.random.default_rng(5)
    mean = np.repeat(rng.integers(-4, 5, (60, 3)) * 0.25, 20, 0) + far
    n = len(mean)
    g = vp.Gaussians(mean.astype(np.float32), np.full((n, 3), 0.05, np.float32),
                     np.tile(np.array([1.0, 0, 0, 0], np.float32), (n, 1)), np.full(n, 2e-3, np.float32),
                     rng.uniform(0.2, 0.95, (n, 3)).astype(np.float32))
    cam = vp.Camera.perspective((far + 0.3, far + 0.2, far - 4.0), (far, far, far), (0.0, 1.0, 0.0), 40.0)
    assert has_8_wide_tree(compare(vp_ctx, g, 290, 240, 16, camera=cam, hg_g=0.0))
