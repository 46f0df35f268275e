"""GPU: small Gaussians seen from far away through a narrow lens, where FP32 rounding of a box test or of a packet's
side planes is as large as the Gaussians: no traversal may lose one that another finds.

Without emission and before a white environment a pixel of one sample is exp(-tau), so the packets' image, the
thread-per-ray query and the megakernel's evaluate the same chords with the same arithmetic, and T is higher only
where a Gaussian was lost.  The reference is the lower T of the megakernel and the warp-per-ray query (each tests
FP32 boxes, too, and may lose some of its own).  Tolerance: 2e-6, the rounding of a sum of up to 16 (FP32 partial
sums of 8 terms in the packets: 8 x 2^-24 x tau e^-tau < 2e-7, FAST exponentials alike).
"""
import math

import numpy as np
import pytest

import volprim_b200 as vp
from volprim_b200._capi import VP_ENGINE_MEGAKERNEL, VP_PRECISION_ACCURATE, VP_PRECISION_FAST
from volprim_b200.emission import render_emission

pytestmark = pytest.mark.gpu

# half the view's height, distance, Gaussians, their sigma over the half height, lens, precision, seed
VIEWS = [(0.01, 3.0, 400, 0.15, False, "accurate", 1), (0.002, 840.0, 1200, 0.025, False, "accurate", 2),
         (0.0014, 1280.0, 97, 0.041, False, "fast", 3), (0.0025, 3400.0, 900, 0.018, False, "fast", 4),
         (0.004, 3500.0, 526, 0.018, False, "accurate", 5), (0.0034, 7700.0, 319, 0.037, False, "accurate", 6),
         (0.0094, 6000.0, 1293, 0.035, True, "accurate", 7), (0.0014, 5900.0, 781, 0.085, True, "fast", 8),
         (0.011, 14700.0, 599, 0.019, False, "fast", 9), (0.0038, 29000.0, 1024, 0.116, True, "fast", 10)]


@pytest.fixture(scope="module", params=VIEWS, ids=lambda v: f"{v[1]:g}{'-ortho' if v[4] else ''}")
def view(request, vp_ctx):
    half, distance, n, size, ortho, precision, seed = request.param
    w, h = 288, 192  # 55,296 rays: packets (the other form's limit is 45,056 here), and a thread on each ray
    rng = np.random.default_rng(seed)
    sigma = half * size
    v = rng.normal(size=3)
    eye = tuple(float(x) for x in v / np.linalg.norm(v) * distance)
    mean = rng.uniform(-half, half, (n, 3)).astype(np.float32)
    g = vp.Gaussians(mean, np.full((n, 3), sigma, np.float32), np.tile(np.array([1.0, 0, 0, 0], np.float32), (n, 1)),
                     np.full(n, 0.7 * sigma ** 2 * 2 * math.pi, np.float32))
    cam = (vp.Camera.orthographic_camera(eye, (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 2 * half) if ortho else
           vp.Camera.perspective(eye, (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), math.degrees(2 * math.atan(half / distance))))
    cfg = vp.Config(num_samples_per_pixel=1, image_width=w, image_height=h, seed=4, precision=precision)
    sc = vp.Scene(vp_ctx, g, 1.0)
    py, px = np.divmod(np.arange(w * h, dtype=np.uint32), np.uint32(w))
    o, d = vp_ctx.camera_rays(cam, cfg, px, py, np.zeros(w * h, np.uint32))
    prec = VP_PRECISION_ACCURATE if precision == "accurate" else VP_PRECISION_FAST
    ref = np.minimum(sc.transmittance(o, d, precision=prec, engine=VP_ENGINE_MEGAKERNEL),
                     sc.transmittance_static(o, d, precision=prec)).astype(np.float64)
    assert (ref < 0.9).mean() > 0.02
    yield sc, cam, cfg, o, d, prec, ref
    sc.close()


def test_packets_lose_none(vp_ctx, view):
    sc, cam, cfg, _, _, _, ref = view
    env = vp.Environment(vp_ctx, constant=(1.0, 1.0, 1.0))
    img = render_emission(sc, env, cam, cfg)[..., 0].astype(np.float64).reshape(-1)
    env.close()
    lost = img - ref > 2e-6
    assert not lost.any(), (int(lost.sum()), float((img - ref).max()))


def test_thread_per_ray_loses_none(view):
    sc, _, _, o, d, prec, ref = view
    got = sc.transmittance(o, d, precision=prec).astype(np.float64)
    lost = got - ref > 2e-6
    assert not lost.any(), (int(lost.sum()), float((got - ref).max()))
