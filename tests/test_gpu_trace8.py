"""GPU: the thread-per-ray stages over the compressed 8-wide BVH (wavefront engine) against the warp engine,
which traverses the BVH32 one path a warp.

Both engines take the same samples, evaluate the same chords with the same arithmetic and carry their
sums in FP64 rounded once, so a pixel differs only where a transmittance reaches MAX_OPTICAL_DEPTH in
one order of summation and not in the other (T below 1e-38), or where a sum lies within 1e-16 of a
rounding boundary.  Hence: every pixel within 1e-5 of the image's mean.
"""
import math

import numpy as np
import pytest

import volprim_b200 as vp
from volprim_b200 import scenes

pytestmark = pytest.mark.gpu

W, H = 409, 281  # 114,929 paths: more than one refill of every warp; the tail kernel takes the last 65,536


def gaussians(n, seed, layout="box", mixed=True):
    rng = np.random.default_rng(seed)
    scale = np.exp(rng.normal(math.log(0.1), 0.5, (n, 3)))
    mean = rng.uniform(-0.6, 0.6, (n, 3))
    if layout == "nested":      # a chain: deeper than the 8-wide tree's limit, so the warp queries run
        scale = np.repeat((0.01 * 1.003 ** np.arange(n))[:, None], 3, 1)
        mean = np.zeros((n, 3))
    elif layout == "same":      # identical boxes
        scale, mean = np.full((n, 3), 0.2), np.full((n, 3), 0.1)
    elif layout == "spread":    # extents from 1e-4 to 1e2 in one tree
        scale = np.exp(rng.uniform(math.log(3e-5), math.log(30.0), (n, 1))) * np.exp(rng.normal(0, 0.3, (n, 3)))
    elif layout == "plate":     # thin in one axis, aligned with it
        scale = np.stack([np.full(n, 0.1), np.full(n, 1e-5), np.full(n, 0.1)], 1)
        mean[:, 1] = 0.25
    quat = scenes.uniform_quaternions(rng, n) if layout != "plate" else np.tile(np.array([1.0, 0, 0, 0]), (n, 1))
    dens = np.exp(rng.normal(-1.0, 0.5, n)) * (8.0 / max(n, 8)) * (scale.prod(1) / 1e-3) ** (2.0 / 3.0)
    albedo = rng.uniform(0.2, 0.95, (n, 3)) if mixed else np.tile(np.array([0.9, 0.8, 0.7]), (n, 1))
    return vp.Gaussians(*(a.astype(np.float32) for a in (mean, scale, quat, dens, albedo)))


def images(ctx, g, sigma=1.0, camera=None, **kw):
    sc = vp.Scene(ctx, g, sigma)
    env = vp.Environment(ctx, rgb=scenes.procedural_env(64, 32, sun_radiance=50.0, sun_radius_deg=8.0))
    out = {}
    for engine in ("wavefront", "warp"):
        cfg = vp.Config(num_samples_per_pixel=1, image_width=W, image_height=H, seed=5, engine=engine, max_bounces=16,
                        rr_depth=4, **kw)
        out[engine] = vp.Renderer(cfg, sc, camera or scenes.negz_camera(3.0, 40.0), env=env, ctx=ctx).render()[..., :3]
    sc.close()
    return out["wavefront"], out["warp"]


def check(a, b):
    assert np.isfinite(a).all() and b.mean() > 1e-3
    assert np.abs(a - b).max() <= 1e-5 * b.mean(), (np.abs(a - b).max(), np.mean(a != b))


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 24, 25, 64, 65, 3000])
@pytest.mark.parametrize("mixed", [False, True])
def test_sizes(vp_ctx, n, mixed):
    check(*images(vp_ctx, gaussians(n, n, mixed=mixed), hg_g=0.6))


@pytest.mark.parametrize("w, h", [(1, 1), (3, 1), (31, 3), (67, 41), (211, 250)])
@pytest.mark.parametrize("mixed", [False, True])
def test_tail(vp_ctx, monkeypatch, w, h, mixed):
    """Images whose paths all go to the tail after their first bounce: from one path to 22 a warp."""
    monkeypatch.setitem(globals(), "W", w)
    monkeypatch.setitem(globals(), "H", h)
    check(*images(vp_ctx, gaussians(400, 12, mixed=mixed), sigma=2.0, hg_g=0.3, camera=scenes.negz_camera(1.2, 30.0)))


@pytest.mark.parametrize("layout", ["nested", "same", "spread", "plate"])
def test_layouts(vp_ctx, layout):
    check(*images(vp_ctx, gaussians(600, 3, layout), hg_g=0.0))


@pytest.mark.parametrize("nee", ["mis", "phase", "ris", "none"])
@pytest.mark.parametrize("precision", ["fast", "accurate"])
def test_estimators(vp_ctx, nee, precision):
    check(*images(vp_ctx, gaussians(500, 9), sigma=3.0, nee=nee, precision=precision, hg_g=0.85))


def test_camera_inside_and_axis_aligned_rays(vp_ctx):
    """An orthographic camera along an axis (two direction components 0), from inside the cloud."""
    cam = vp.Camera.orthographic_camera((0.0, 0.0, -0.2), (0.0, 0.0, 1.0), (0.0, 1.0, 0.0), 1.0)
    check(*images(vp_ctx, gaussians(800, 4), camera=cam, hg_g=0.0))


def test_empty_scene(vp_ctx):
    g = vp.Gaussians(np.zeros((0, 3), np.float32), np.zeros((0, 3), np.float32), np.zeros((0, 4), np.float32),
                     np.zeros(0, np.float32))
    check(*images(vp_ctx, g))


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1000, 114_700])
def test_transmittance_batches(vp_ctx, n):
    """vp_transmittance (thread per ray) against vp_transmittance_static (warp per ray over the BVH32)."""
    sc = vp.Scene(vp_ctx, gaussians(1500, 21), 0.2)
    rng = np.random.default_rng(22)
    o = np.where((np.arange(n) % 2 == 0)[:, None], rng.normal(0, 2.0, (n, 3)), rng.uniform(-0.5, 0.5, (n, 3)))
    d = rng.normal(0, 1, (n, 3))
    d[::7, 0] = 0.0  # axis-parallel components
    d = d / np.linalg.norm(d, axis=1, keepdims=True)
    o, d = o.astype(np.float32), d.astype(np.float32)
    for precision in (vp.VP_PRECISION_FAST, vp.VP_PRECISION_ACCURATE):
        got = sc.transmittance(o, d, precision=precision)
        want = np.concatenate([sc.transmittance_static(o[k:k + 50_000], d[k:k + 50_000], precision=precision)
                               for k in range(0, n, 50_000)])
        assert n < 1000 or ((want < 0.9).sum() > n // 100 and (want > 0.99).sum() > n // 100)
        assert np.abs(got - want).max() <= 1e-7, np.abs(got - want).max()
    sc.close()


def test_served_requests_match_renders(vp_ctx):
    """Two scenes -- one of one albedo, one mixed -- and a pool of path slots above the threshold: every request
    equals its own render up to the order of its pixel sums."""
    from volprim_b200 import serving
    env = vp.Environment(vp_ctx, rgb=scenes.procedural_env(64, 32, sun_radiance=50.0, sun_radius_deg=8.0))
    scs = [vp.Scene(vp_ctx, gaussians(700, 31 + k, mixed=bool(k))) for k in range(2)]
    server = serving.Server(vp_ctx, path_slots=1 << 18)
    for s in scs:
        server.add_scene(s, env)
    reqs = []
    for k, (w, h, spp) in enumerate([(300, 250, 2), (301, 203, 2), (64, 64, 4), (257, 129, 3)]):
        cfg = vp.Config(num_samples_per_pixel=spp, image_width=w, image_height=h, seed=k, hg_g=0.3, max_bounces=12,
                        rr_depth=12, precision="fast")
        cam = serving.random_camera(np.random.default_rng(k), 3.0)
        reqs.append((server.submit(k % 2, cam, cfg), k % 2, cam, cfg))
    left = len(reqs)
    while left:
        server.step()
        left -= len(server.poll())
    for rid, k, cam, cfg in reqs:
        got = server.result(rid)[..., :3]
        want = vp.Renderer(cfg, scs[k], cam, env=env, ctx=vp_ctx).render()[..., :3]
        assert np.abs(got - want).max() <= 1e-5 * want.max() + 1e-6
    server.close()
    for s in scs:
        s.close()


def test_nodes_below_the_distance_rounding(vp_ctx):
    """A node far smaller than an ulp of the ray's distance to it: all its planes round to one distance, those of
    its unused slots too, and only its three Gaussians may be met."""
    c = np.array([[0.0, 0.0, 0.0], [2e-8, 0.0, 0.0], [0.0, 2e-8, 1e-8]], np.float32)
    g = vp.Gaussians(c, np.full((3, 3), 1e-8, np.float32), np.tile(np.array([1.0, 0, 0, 0], np.float32), (3, 1)),
                     np.full(3, 1e-16, np.float32), np.full((3, 3), 0.5, np.float32))
    cam = vp.Camera.orthographic_camera((0.0, 0.0, -100.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 2e-7)
    check(*images(vp_ctx, g, camera=cam, hg_g=0.0))
