"""GPU: the emission image and its adjoint in both their forms -- a warp on each ray for images of few rays,
packets of rays above that -- at the edges of their tilings (one sample to more than a warp's, images that
are no multiple of a tile, every block size), against the FP64 oracle over all (ray, Gaussian) pairs.  Tolerances are those of test_gpu_emission.py: each pixel
within 1e-4 max(|L64|, 1e-2), each parameter group within 1e-3 relative (L2) -- over the Gaussians that no
ray grazes: tau has a square-root kink at d2 = 9, so its derivative is as uncertain as d2's FP32 rounding
(about 1e-6) over 9 - d2."""
import math

import numpy as np
import pytest
import torch

import emission_oracle as E
import oracle as O
import volprim_b200 as vp
from volprim_b200 import scenes
from volprim_b200.emission import render_emission, render_emission_backward

pytestmark = pytest.mark.gpu

CAMERAS = {"outside": vp.Camera.perspective((0.4, 0.3, -3.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 40.0),
           "inside": vp.Camera.perspective((0.05, 0.0, -0.1), (0.3, 0.2, 1.0), (0.0, 1.0, 0.0), 70.0),
           "ortho": vp.Camera.orthographic_camera((0.0, 0.2, -3.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 1.8)}


def scene_of(n, seed, size=0.12):
    rng = np.random.default_rng(seed)
    mean = rng.uniform(-0.6, 0.6, (n, 3)).astype(np.float32)
    log_scale = rng.normal(math.log(size), 0.4, (n, 3)).astype(np.float32)
    dens = (np.exp(rng.normal(0.0, 0.5, n)) * 4.0 / n).astype(np.float32)
    g = vp.Gaussians(mean, log_scale, scenes.uniform_quaternions(rng, n), dens, None, scale_is_log=True)
    return g, rng.uniform(0.0, 1.0, (n, 3)).astype(np.float32)


def check(ctx, g, em, cam, w, h, spp, seed=3, crop=None):
    x0, y0, cw, ch = crop or (0, 0, w, h)  # the pixels compared, and the only ones with an upstream gradient
    n = g.count
    cfg = vp.Config(num_samples_per_pixel=spp, image_width=w, image_height=h, seed=seed, precision="fast")
    sc = vp.Scene(ctx, g, 1.0)
    sc.set_emission(em)
    env = vp.Environment(ctx, constant=(0.7, 0.8, 0.9))
    img = render_emission(sc, env, cam, cfg)[..., :3].astype(np.float64)
    img = img[y0:y0 + ch, x0:x0 + cw]

    px, py = np.meshgrid(np.arange(x0, x0 + cw), np.arange(y0, y0 + ch))
    px, py = np.repeat(px.reshape(-1), spp), np.repeat(py.reshape(-1), spp)
    o, d = O.camera_rays(O.camera16(cam, w, h), w, spp, seed, px, py, np.tile(np.arange(spp), cw * ch))
    o, d = torch.tensor(o, dtype=torch.float64), torch.tensor(d, dtype=torch.float64)
    R = len(o)
    p = E.params_from(g, requires_grad=True)
    e = torch.tensor(em, dtype=torch.float64, requires_grad=True)
    ri = torch.arange(R).repeat_interleave(n)
    gi = torch.arange(n).repeat(R)
    S, C = E.ray_sums(p, e, 1.0, o, d, ri, gi, R)
    bg = torch.tensor([0.7, 0.8, 0.9], dtype=torch.float64).expand(R, 3)
    ref = E.radiance(S, C, bg).view(ch, cw, spp, 3).mean(2)
    err = np.abs(img - ref.detach().numpy())
    assert np.abs(ref.detach().numpy() - bg[0].numpy()).max() > 0.05, "the image must see the cloud"
    assert np.all(err <= 1e-4 * np.maximum(np.abs(ref.detach().numpy()), 1e-2)), float(err.max())

    up = np.zeros((h, w, 4), np.float32)
    part = np.random.default_rng(seed).normal(0.0, 1.0, (ch, cw, 4)).astype(np.float32)
    part[::3, ::2, :3] = 0.0  # pixels nothing flows back from
    up[y0:y0 + ch, x0:x0 + cw] = part
    grads = {"mean": np.zeros(3 * n, np.float32), "scale": np.zeros(3 * n, np.float32),
             "quat_wxyz": np.zeros(4 * n, np.float32), "density": np.zeros(n, np.float32),
             "emission": np.zeros(3 * n, np.float32)}
    render_emission_backward(sc, env, cam, cfg, up, grads)
    (ref * torch.tensor(part[..., :3], dtype=torch.float64)).sum().backward()
    want = {"mean": p["mean"].grad, "scale": p["log_scale"].grad, "quat_wxyz": p["quat"].grad,
            "density": p["density"].grad, "emission": e.grad}
    grazed = gi[(9.0 - E.pair_d2(p, o, d, ri, gi)).abs() < 1e-4].unique().numpy()
    assert len(grazed) < n
    for k, v in want.items():
        v, got = v.numpy().reshape(n, -1).copy(), grads[k].reshape(n, -1).copy()
        v[grazed] = got[grazed] = 0.0
        assert np.linalg.norm(got - v) <= 1e-3 * np.linalg.norm(v), (k, np.linalg.norm(got - v) / np.linalg.norm(v))
    env.close()
    sc.close()


@pytest.mark.parametrize("w, h, spp", [(17, 13, 1), (9, 7, 3), (11, 6, 8), (7, 5, 17), (5, 4, 33), (3, 2, 64), (1, 1, 32)])
@pytest.mark.parametrize("camera", list(CAMERAS))
def test_tiles(vp_ctx, w, h, spp, camera):
    if (w, h) == (1, 1) and camera == "inside":
        w, h = 2, 1  # its one pixel spans 70 degrees and sees hardly anything of the cloud's own size
    check(vp_ctx, *scene_of(150, 5), CAMERAS[camera], w, h, spp)


@pytest.mark.parametrize("n", [1, 24, 33])
def test_few_gaussians(vp_ctx, n):
    check(vp_ctx, *scene_of(n, n, 0.3), CAMERAS["outside"], 13, 9, 4)


def test_more_gaussians_than_the_list(vp_ctx):
    """A warp meets more than 512 Gaussians, so the adjoint's second pass traverses again."""
    check(vp_ctx, *scene_of(6000, 8, 0.3), CAMERAS["outside"], 6, 4, 2)


@pytest.mark.parametrize("w, h", [(96, 90), (230, 190)])
def test_block_sizes(vp_ctx, w, h):
    """Enough tiles (1,080 of 8 pixels x 4 samples, 10,925 of 4 x 8) for blocks of 4 and of 2 warps."""
    spp = 4 if w == 96 else 8
    check(vp_ctx, *scene_of(12, 2, 0.15), CAMERAS["outside"], w, h, spp)


# More rays than the form with a warp on each takes (45,056 forward, 67,584 adjoint for a scene this small); the last
# has few enough tiles for blocks of 8 warps.
@pytest.mark.parametrize("w, h, spp", [(263, 259, 1), (151, 150, 3), (93, 91, 8), (67, 60, 17), (47, 44, 33), (37, 29, 64),
                                       (12, 9, 640)])
@pytest.mark.parametrize("camera", list(CAMERAS))
def test_packet_tiles(vp_ctx, w, h, spp, camera):
    check(vp_ctx, *scene_of(12, 2, 0.15), CAMERAS[camera], w, h, spp)


@pytest.mark.parametrize("w, h, spp", [(256, 176, 1), (45057, 1, 1), (352, 192, 1), (67585, 1, 1)])
def test_either_side_of_the_rule(vp_ctx, w, h, spp):
    """The largest image a form takes, and the smallest the next one does, forward (45,056) and adjoint (67,584)."""
    check(vp_ctx, *scene_of(3, 2, 0.3), CAMERAS["ortho"], w, h, spp)


def test_packets_of_more_gaussians_than_the_list(vp_ctx):
    check(vp_ctx, *scene_of(6000, 8, 0.3), CAMERAS["outside"], 190, 180, 2, crop=(92, 88, 6, 4))
