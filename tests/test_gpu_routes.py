"""GPU: routes that the sizes of the other tests do not reach -- short ray batches through scenes large enough for a
thread on each ray, ACCURATE emission packets in blocks of four and eight warps, the two orders of the warp-per-ray
transmittance, and a server with a scene that has no 8-wide tree."""
import numpy as np
import pytest

import test_gpu_emission_packets as P
import test_gpu_few_paths as F
import test_gpu_trace8 as T
import volprim_b200 as vp
from volprim_b200 import scenes, serving

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1000, 30_000])
@pytest.mark.parametrize("precision", [vp.VP_PRECISION_FAST, vp.VP_PRECISION_ACCURATE])
def test_short_batches_by_threads(vp_ctx, n, precision):
    """From 16,384 Gaussians on any batch has a thread on each ray; vp_transmittance_static has a warp.  The same
    chords in FP64 sums rounded once: 1e-7."""
    rng = np.random.default_rng(31)
    k = 20_000
    g = vp.Gaussians(rng.uniform(-0.8, 0.8, (k, 3)).astype(np.float32), np.full((k, 3), 0.03, np.float32),
                     scenes.uniform_quaternions(rng, k).astype(np.float32), np.full(k, 3e-5, np.float32))
    sc = vp.Scene(vp_ctx, g, 1.0)
    assert F.has_8_wide_tree(sc.info())
    o = np.where((np.arange(n) % 2 == 0)[:, None], rng.normal(0, 2.0, (n, 3)), rng.uniform(-0.5, 0.5, (n, 3)))
    d = rng.uniform(-0.5, 0.5, (n, 3)) - o
    d = d / np.linalg.norm(d, axis=1, keepdims=True)
    o, d = o.astype(np.float32), d.astype(np.float32)
    got = sc.transmittance(o, d, precision=precision)
    want = sc.transmittance_static(o, d, precision=precision)
    assert (want < 0.99).mean() > 0.5
    assert np.abs(got - want).max() <= 1e-7, np.abs(got - want).max()
    sc.close()


# more rays than the form with a warp on each takes (54,067 for the ACCURATE adjoint); 2,000 and more tiles: blocks of 4
# warps, 108 tiles: of 8
@pytest.mark.parametrize("w, h, spp", [(263, 259, 1), (93, 91, 8), (12, 9, 640)])
@pytest.mark.parametrize("camera", list(P.CAMERAS))
def test_accurate_packets(vp_ctx, monkeypatch, w, h, spp, camera):
    config = vp.Config
    monkeypatch.setattr(vp, "Config", lambda **kw: config(**{**kw, "precision": "accurate"}))
    P.check(vp_ctx, *P.scene_of(12, 2, 0.15), P.CAMERAS[camera], w, h, spp)


@pytest.mark.parametrize("make, sigma", [(scenes.stress_gaussians, 1.0), (scenes.showcase_gaussians, 7.5)])
def test_tau_orders_of_the_warp_queries(vp_ctx, make, sigma):
    """The order of a node's children changes only when a ray reaches MAX_OPTICAL_DEPTH and the order of FP64 sums:
    1e-7 in T; an image's pixels within 1e-5 of its mean."""
    g = make(30_000, 3)
    sc = {k: vp.Scene(vp_ctx, g, sigma, tau_order=k) for k in ("lane", "nearest")}
    rng = np.random.default_rng(11)
    n = 20_000
    o = rng.normal(size=(n, 3))
    o = np.where((np.arange(n) % 2 == 0)[:, None], g.mean[rng.choice(len(g.density), n)],
                 3.0 * o / np.linalg.norm(o, axis=1, keepdims=True))
    d = rng.uniform(-0.6, 0.6, (n, 3)) - o
    d = d / np.linalg.norm(d, axis=1, keepdims=True)
    o, d = o.astype(np.float32), d.astype(np.float32)
    for precision in (vp.VP_PRECISION_FAST, vp.VP_PRECISION_ACCURATE):
        a, b = (sc[k].transmittance_static(o, d, precision=precision) for k in ("lane", "nearest"))
        assert (a < 0.99).sum() > 1000
        assert np.abs(a - b).max() <= 1e-7
    env = vp.Environment(vp_ctx, rgb=scenes.procedural_env(64, 32, sun_radiance=50.0, sun_radius_deg=8.0))
    cfg = vp.Config(num_samples_per_pixel=4, image_width=64, image_height=48, seed=3, hg_g=0.0, max_bounces=16, rr_depth=16,
                    engine="warp", precision="fast")
    a, b = (vp.Renderer(cfg, sc[k], scenes.negz_camera(), env=env, ctx=vp_ctx).render()[..., :3] for k in ("lane", "nearest"))
    T.check(a, b)
    env.close()
    for s in sc.values():
        s.close()


@pytest.mark.parametrize("other", ["nested", "overlapping", "empty"])
@pytest.mark.parametrize("precision", ["fast", "accurate"])
def test_server_with_a_scene_without_the_8_wide_tree(vp_ctx, other, precision):
    """One such scene sends all of the server's to the warp queries; every request equals its own render up to the
    order of its pixel sums."""
    none = vp.Gaussians(np.zeros((0, 3), np.float32), np.zeros((0, 3), np.float32), np.zeros((0, 4), np.float32),
                        np.zeros(0, np.float32))
    second = {"nested": lambda: T.gaussians(600, 3, "nested"), "overlapping": lambda: F.box(300, 11, 0.4, True),
              "empty": lambda: none}[other]()
    env = vp.Environment(vp_ctx, rgb=scenes.procedural_env(64, 32, sun_radiance=50.0, sun_radius_deg=8.0))
    scs = [vp.Scene(vp_ctx, T.gaussians(700, 31)), vp.Scene(vp_ctx, second)]
    assert other == "empty" or not F.has_8_wide_tree(scs[1].info())
    server = serving.Server(vp_ctx, path_slots=1 << 16, precision=precision)
    for s in scs:
        server.add_scene(s, env)
    reqs = []
    for k, (w, h, spp) in enumerate([(100, 80, 2), (101, 63, 2), (64, 64, 1), (57, 29, 3)]):
        cfg = vp.Config(num_samples_per_pixel=spp, image_width=w, image_height=h, seed=k, hg_g=0.3, max_bounces=12,
                        rr_depth=12, precision=precision)
        cam = serving.random_camera(np.random.default_rng(k), 3.0)
        reqs.append((server.submit(k % 2, cam, cfg), k % 2, cam, cfg))
    left = len(reqs)
    while left:
        server.step()
        left -= len(server.poll())
    for rid, k, cam, cfg in reqs:
        got = server.result(rid)[..., :3]
        want = vp.Renderer(cfg, scs[k], cam, env=env, ctx=vp_ctx).render()[..., :3]
        assert want.mean() > 1e-3
        assert np.abs(got - want).max() <= 1e-5 * want.max() + 1e-6
    server.close()
    env.close()
    for s in scs:
        s.close()
