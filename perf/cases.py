"""What the framework's speed is measured on: the calls a user makes, over the range of scenes, images and
batches they are made with.

    listed()            the fixed cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) the scene, environment, rays or parameters a program holds before the call (on the GPU)
    run(state)          one call through the public interface, and what it returns
    work(case)          the bytes and floating-point operations the call cannot do without
    exact(case, seed)   the closed-form results in 64 bits, where the call computes one

Scenes follow the distributions of volprim_b200.scenes (the 256-Gaussian absorption scene, the value-noise
cloud, the 16-cluster stress scene, the emission and serving workloads), drawn with torch on the GPU.

Images of more than some 30,000 paths stop at the depth where Russian roulette starts (max_bounces =
rr_depth = 12): beyond it a last-bit change of a throughput can end a path one bounce earlier, so two correct
renders of the same samples differ by whole paths.  Smaller images run to the configured depth with roulette.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "cuda-volprim_b200"))

import volprim_b200 as vp  # noqa: E402
from volprim_b200 import emission as vpe  # noqa: E402
from volprim_b200 import serving  # noqa: E402
from volprim_b200.autograd import render_emission_images  # noqa: E402

CHORD_FLOPS = 111   # one closed-form chord: whitening, closest approach, erf difference, exponential
RECORD_BYTES = 56   # mean, scale, quaternion, density and albedo of one Gaussian

_ctx = None


def context():
    """The program's one device context."""
    global _ctx
    if _ctx is None:
        _ctx = vp.Context(0)
    return _ctx


# ---- cases ---------------------------------------------------------------------------------
def _render(name, scene, n, width, height, spp, depth, nee="mis", g=0.0, env="procedural", precision="auto",
            filt=0.0, clamp=0.0):
    return {"name": name, "kind": "render", "scene": scene, "n": n, "width": width, "height": height, "spp": spp,
            "depth": depth, "nee": nee, "g": g, "env": env, "precision": precision, "filter": filt, "clamp": clamp}


def listed():
    return [
        # the absorption-only image of the 256-Gaussian scene: a call of well under a millisecond, where launches
        # and host work count
        _render("absorption_256", "uniform", 256, 128, 128, 16, 128, env="white"),
        # one 16-sample batch of the 500k-Gaussian showcase: what a production render spends its time on
        _render("showcase_500k", "cloud", 500_000, 512, 512, 16, 12),
        # an interactive preview: one sample a pixel of a small image, all 64 bounces
        _render("preview_64", "cloud", 50_000, 64, 64, 1, 64),
        # two million Gaussians in dense overlapping clusters, an image that is no multiple of anything
        _render("stress_2m", "clusters", 2_000_000, 641, 427, 8, 12),
        # the other estimator with everything on: RIS, anisotropic phase, pixel filter, firefly clamp, odd sizes
        _render("ris_filtered", "cloud", 100_000, 333, 217, 5, 12, nee="ris", g=0.85, filt=0.5, clamp=20.0),
        # a program that starts, loads a scene and an HDR map from host memory, renders and exits
        {"name": "load_and_render", "kind": "load", "n": 250_000, "env_width": 1024, "env_height": 512,
         "width": 96, "height": 54, "spp": 4},
        # transmittance of a batch of device-resident rays through the cloud (a plug-in's shadow query)
        {"name": "transmittance_batch", "kind": "transmittance", "scene": "cloud", "n": 100_000, "rays": 250_007,
         "precision": "fast", "host": False},
        # a handful of host rays through a small scene: all latency
        {"name": "transmittance_few", "kind": "transmittance", "scene": "uniform", "n": 1000, "rays": 1023,
         "precision": "accurate", "host": True},
        # albedo and overlap counts at points of the cloud (baking to a grid)
        {"name": "albedo_points", "kind": "albedo", "scene": "cloud", "n": 100_000, "points": 50_001},
        # the differentiable image, forward only (a validation view during a fit)
        {"name": "emission_view", "kind": "emission", "n": 100_000, "width": 256, "height": 256, "spp": 8,
         "precision": "fast"},
        # one optimisation step of the fit: scene build, forward and adjoint of two views, all gradients
        {"name": "emission_step", "kind": "train", "n": 100_000, "width": 160, "height": 120, "spp": 8, "views": 2,
         "precision": "fast"},
        # a burst of mixed requests served together from two resident scenes
        {"name": "serve_burst", "kind": "serve", "n0": 50_000, "n1": 100_000, "requests": 16, "depth": 12},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render"] * 5 + ["load", "transmittance", "transmittance", "albedo", "emission", "train", "serve"])
    if kind == "render":
        scene = rng.choice(["cloud", "cloud", "clusters", "uniform"])
        n = _log_int(rng, 200, 5000) if scene == "uniform" else _log_int(rng, 10_000, 500_000)
        small = rng.random() < 0.4
        if small:
            w, h, spp = rng.randint(31, 120), rng.randint(31, 90), rng.randint(1, 2)
        else:
            w, h, spp = rng.randint(120, 520), rng.randint(90, 400), rng.randint(1, 16)
        c = _render("", scene, n, w, h, spp, rng.choice([32, 64, 128]) if small else rng.choice([8, 12]),
                    nee=rng.choice(["mis", "mis", "ris", "phase", "none"]), g=rng.choice([0.0, 0.6, 0.85]),
                    env="white" if scene == "uniform" else "procedural",
                    precision=rng.choice(["auto", "auto", "auto", "accurate"]) if scene != "uniform" else "auto",
                    filt=rng.choice([0.0, 0.0, 0.5]))
        del c["name"]
        return c
    if kind == "load":
        return {"kind": kind, "n": _log_int(rng, 20_000, 400_000), "env_width": rng.choice([511, 1000, 1024, 2048]),
                "env_height": rng.choice([255, 500, 512, 1024]), "width": rng.randint(33, 100),
                "height": rng.randint(33, 70), "spp": rng.randint(1, 4)}
    if kind == "transmittance":
        scene = rng.choice(["cloud", "clusters", "uniform"])
        n = _log_int(rng, 200, 5000) if scene == "uniform" else _log_int(rng, 10_000, 100_000)
        return {"kind": kind, "scene": scene, "n": n, "rays": _log_int(rng, 500, 250_000),
                "precision": rng.choice(["fast", "accurate"]), "host": rng.random() < 0.5}
    if kind == "albedo":
        return {"kind": kind, "scene": rng.choice(["cloud", "clusters"]), "n": _log_int(rng, 10_000, 100_000),
                "points": _log_int(rng, 500, 50_000)}
    if kind == "emission":
        return {"kind": kind, "n": _log_int(rng, 5000, 100_000), "width": rng.randint(40, 256),
                "height": rng.randint(40, 256), "spp": rng.randint(1, 8),
                "precision": rng.choice(["fast", "fast", "accurate"])}
    if kind == "train":
        return {"kind": kind, "n": _log_int(rng, 5000, 100_000), "width": rng.randint(40, 160),
                "height": rng.randint(40, 120), "spp": rng.randint(1, 8), "views": rng.randint(1, 2),
                "precision": "fast"}
    return {"kind": "serve", "n0": _log_int(rng, 10_000, 100_000), "n1": _log_int(rng, 10_000, 100_000),
            "requests": rng.randint(2, 16), "depth": rng.choice([8, 12])}


# ---- scenes, drawn on the GPU ----------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float32)


def _normal(g, mu, sigma, *shape):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32) * sigma + mu


def _quats(g, n):
    u1, u2, u3 = _rand(g, 3, n)
    a, b, t = (1.0 - u1).sqrt(), u1.sqrt(), 2.0 * math.pi
    return torch.stack([b * torch.cos(t * u3), a * torch.sin(t * u2), a * torch.cos(t * u2), b * torch.sin(t * u3)], 1)


def _value_noise(g, x):
    """Three octaves of smoothstep-trilinear lattice noise over the 2 x 1 x 1 box."""
    total, amp, norm = 0.0, 1.0, 0.0
    u = (x - torch.tensor([-1.0, -0.5, -0.5], device="cuda")) / torch.tensor([2.0, 1.0, 1.0], device="cuda")
    for o in range(3):
        c = torch.tensor([8 << o, 4 << o, 4 << o], device="cuda")
        lat = _rand(g, (8 << o) + 1, (4 << o) + 1, (4 << o) + 1)
        y = u.clamp(0, 1) * c
        i = torch.minimum(y.floor().long(), c - 1)
        f = y - i
        f = f * f * (3.0 - 2.0 * f)
        acc = 0.0
        for dx in (0, 1):
            for dy in (0, 1):
                for dz in (0, 1):
                    w = ((f[:, 0] if dx else 1 - f[:, 0]) * (f[:, 1] if dy else 1 - f[:, 1])
                         * (f[:, 2] if dz else 1 - f[:, 2]))
                    acc = acc + w * lat[i[:, 0] + dx, i[:, 1] + dy, i[:, 2] + dz]
        total, norm, amp = total + amp * acc, norm + amp, amp * 0.5
    return total / norm


def _gaussians(scene, n, seed):
    """(Gaussians of CUDA tensors, sigma multiplier)."""
    g = _gen(seed)
    if scene == "uniform":  # absorption_256's distributions
        mean, scale = _rand(g, n, 3) * 2 - 1, _normal(g, math.log(0.1), 0.4, n, 3).exp()
        density, albedo, sigma = _normal(g, math.log(5.0), 0.5, n).exp(), torch.zeros((n, 3), device="cuda"), 1.0
    elif scene == "clusters":  # stress_2m's
        centres = _rand(g, 16, 3) * 1.4 - 0.7
        mean = centres[torch.randint(0, 16, (n,), generator=g, device="cuda")] + _normal(g, 0.0, 0.15, n, 3)
        scale = _normal(g, math.log(0.05), 0.3, n, 3).exp()
        density, albedo, sigma = _normal(g, math.log(2.0), 0.5, n).exp(), torch.full((n, 3), 0.8, device="cuda"), 1.0
    else:  # showcase_500k's: means where a value-noise field exceeds a threshold
        kept, have = [], 0
        state = int(seed) + 7919
        while have < n:
            x = (_rand(g, max(4 * (n - have), 4096), 3) - 0.5) * torch.tensor([2.0, 1.0, 1.0], device="cuda")
            x = x[_value_noise(_gen(state), x) > 0.55]
            kept.append(x)
            have += x.shape[0]
        mean = torch.cat(kept)[:n]
        scale = _normal(g, math.log(0.02), 0.5, n, 3).exp()
        density, albedo, sigma = _normal(g, 0.0, 0.7, n).exp(), torch.full((n, 3), 0.9, device="cuda"), 7.5
    return vp.Gaussians(mean.contiguous(), scale, _quats(g, n), density, albedo), sigma


def _env_image(width, height):
    """volprim_b200.scenes.procedural_env, on the GPU."""
    polar = ((torch.arange(height, device="cuda") + 0.5) / height * math.pi)[:, None]
    theta = (((torch.arange(width, device="cuda") + 0.5) / width - 0.5) * 2 * math.pi)[None, :]
    dx, dy, dz = polar.sin() * theta.cos(), polar.cos().expand(height, width), polar.sin() * theta.sin()
    up = dy.clamp(0, 1)
    sky = torch.stack([0.35 + 0.25 * (1 - up), 0.55 + 0.25 * (1 - up), 0.95 - 0.1 * up], -1)
    img = torch.where((dy >= 0)[..., None], sky, torch.tensor([0.08, 0.07, 0.06], device="cuda"))
    s = np.array([0.7197, 0.4530, 0.5261])
    s = s / np.linalg.norm(s)
    sun = dx * s[0] + dy * s[1] + dz * s[2] >= math.cos(math.radians(0.5))
    img[sun] = torch.tensor([1e4, 9.5e3, 8.5e3], device="cuda")
    return img.contiguous()


def _camera(seed, vfov=40.0):
    """A pinhole camera at distance 3.5 from the origin, looking at it (the serving workload's)."""
    return serving.random_camera(np.random.default_rng(seed), 3.5, vfov)


def _config(case, seed):
    return vp.Config(num_samples_per_pixel=case["spp"], image_width=case["width"], image_height=case["height"],
                     seed=int(seed) & 0x7FFFFFFF, max_bounces=case.get("depth", 128), rr_depth=12,
                     hg_g=case.get("g", 0.0), nee=case.get("nee", "mis"), precision=case.get("precision", "auto"),
                     pixel_filter_stddev=case.get("filter", 0.0), firefly_clamp_luminance=case.get("clamp", 0.0))


def _ray_arrays(n, seed):
    """Rays through the scenes' box: half from the radius-3.5 sphere towards a point of the box, half from inside."""
    g = _gen(seed + 1)
    box = torch.tensor([1.0, 0.5, 0.5], device="cuda")
    aim, inside = (_rand(g, n, 3) * 2 - 1) * box, (_rand(g, n, 3) * 2 - 1) * box
    out = torch.nn.functional.normalize(_normal(g, 0, 1, n, 3), dim=1) * 3.5
    o = torch.where((torch.arange(n, device="cuda") % 2 == 0)[:, None], out, inside)
    d = torch.where((torch.arange(n, device="cuda") % 2 == 0)[:, None], aim - o, _normal(g, 0, 1, n, 3))
    return o.contiguous(), torch.nn.functional.normalize(d.double(), dim=1).float().contiguous()


def _points(gauss, k, seed):
    """Points spread around the Gaussian centres."""
    g = _gen(seed + 2)
    at = torch.randint(0, gauss.mean.shape[0], (k,), generator=g, device="cuda")
    return (gauss.mean[at] + _normal(g, 0, 0.02, k, 3)).cpu().numpy()


def _emission_params(case, seed):
    gauss, sigma = _gaussians("cloud", case["n"], seed)
    e = _rand(_gen(seed + 3), case["n"], 3)
    return [gauss.mean, gauss.scale.log(), gauss.quat_wxyz, gauss.density, e], sigma


def _requests(case, seed):
    """The serving workload's request mix; the seed draws the cameras and the sample streams."""
    trace = serving.make_trace(2024, case["requests"], 0.0, 2, resolutions=(64, 128, 256), spps=(1, 4, 16),
                               max_bounces=case["depth"])
    for i, r in enumerate(trace):
        r.camera, r.config.seed = _camera(1000 * seed + i), (seed + i) & 0x7FFFFFFF
    return trace


def _target(case, seed):
    return _rand(_gen(seed + 4), case["views"], case["height"], case["width"], 3)


# ---- the calls -----------------------------------------------------------------------------
def prepare(case, seed):
    ctx = context()
    kind = case["kind"]
    if kind == "render":
        gauss, sigma = _gaussians(case["scene"], case["n"], seed)
        env = (vp.Environment(ctx, constant=(1.0, 1.0, 1.0)) if case["env"] == "white"
               else vp.Environment(ctx, rgb=_env_image(2048, 1024)))
        r = vp.Renderer(_config(case, seed), vp.Scene(ctx, gauss, sigma), _camera(seed), env=env, ctx=ctx)
        return {"kind": kind, "renderer": r,
                "out": torch.empty((case["height"], case["width"], 4), dtype=torch.float32, device="cuda")}
    if kind == "load":
        gauss, sigma = _gaussians("cloud", case["n"], seed)
        host = vp.Gaussians(*(t.cpu().numpy() for t in (gauss.mean, gauss.scale, gauss.quat_wxyz, gauss.density,
                                                         gauss.albedo)))
        return {"kind": kind, "gaussians": host, "sigma": sigma, "camera": _camera(seed),
                "env": _env_image(case["env_width"], case["env_height"]).cpu().numpy(),
                "config": _config({**case, "depth": 64}, seed)}
    if kind == "transmittance":
        gauss, sigma = _gaussians(case["scene"], case["n"], seed)
        o, d = _ray_arrays(case["rays"], seed)
        if case["host"]:
            o, d = o.cpu().numpy(), d.cpu().numpy()
        return {"kind": kind, "scene": vp.Scene(ctx, gauss, sigma), "o": o, "d": d,
                "precision": vp.VP_PRECISION_FAST if case["precision"] == "fast" else vp.VP_PRECISION_ACCURATE}
    if kind == "albedo":
        gauss, sigma = _gaussians(case["scene"], case["n"], seed)
        gauss.albedo = _rand(_gen(seed + 5), case["n"], 3)
        return {"kind": kind, "scene": vp.Scene(ctx, gauss, sigma), "points": _points(gauss, case["points"], seed)}
    if kind == "emission":
        (mean, log_scale, quat, density, e), sigma = _emission_params(case, seed)
        sc = vp.Scene(ctx, vp.Gaussians(mean, log_scale, quat, density, None, scale_is_log=True), sigma)
        sc.set_emission(e)
        return {"kind": kind, "scene": sc, "env": vp.Environment(ctx, constant=(1.0, 1.0, 1.0)),
                "camera": _camera(seed), "config": _config(case, seed),
                "out": torch.empty((case["height"], case["width"], 4), dtype=torch.float32, device="cuda")}
    if kind == "train":
        params, sigma = _emission_params(case, seed)
        return {"kind": kind, "params": [p.requires_grad_() for p in params], "sigma": sigma,
                "env": vp.Environment(ctx, constant=(1.0, 1.0, 1.0)), "config": _config(case, seed),
                "cameras": [_camera(seed + k) for k in range(case["views"])], "target": _target(case, seed)}
    assert kind == "serve"
    env = vp.Environment(ctx, rgb=_env_image(2048, 1024))
    scenes = [vp.Scene(ctx, *_gaussians("cloud", case[k], seed + i)) for i, k in enumerate(("n0", "n1"))]
    server = serving.Server(ctx, schedule="srpt")
    for sc in scenes:
        server.add_scene(sc, env)
    trace = _requests(case, seed)
    outs = [torch.empty((r.config.image_height, r.config.image_width, 4), dtype=torch.float32, device="cuda")
            for r in trace]
    return {"kind": kind, "server": server, "trace": trace, "outs": outs, "keep": (scenes, env)}


def run(state):
    kind = state["kind"]
    if kind == "render":
        return state["renderer"].render(out=state["out"])
    if kind == "load":
        r = vp.Renderer(state["config"], state["gaussians"], state["camera"], env=state["env"],
                        sigma_multiplier=state["sigma"], ctx=context())
        return r.render()
    if kind == "transmittance":
        return state["scene"].transmittance(state["o"], state["d"], precision=state["precision"])
    if kind == "albedo":
        rgb, count = state["scene"].albedo_at(state["points"])
        return {"rgb": rgb, "overlap": count.astype(np.int64)}
    if kind == "emission":
        return vpe.render_emission(state["scene"], state["env"], state["camera"], state["config"], out=state["out"])
    if kind == "train":
        images = render_emission_images(*state["params"], state["cameras"], state["config"], state["env"],
                                        state["sigma"])
        grads = torch.autograd.grad(((images - state["target"]) ** 2).sum(), state["params"])
        return {"images": images.detach(), **dict(zip(("mean", "log_scale", "quat", "density", "emission"), grads))}
    server, left = state["server"], len(state["trace"])
    for r, out in zip(state["trace"], state["outs"]):
        server.submit(r.scene_id, r.camera, r.config, out)
    while left:
        server.step()
        for rid in server.poll():
            server.result(rid)
            left -= 1
    return state["outs"]


# ---- what a call cannot do without -----------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("render", "load"):
        px = case["width"] * case["height"]
        env = 0 if case.get("env") == "white" else (case.get("env_width", 2048) * case.get("env_height", 1024) * 12)
        # a path has at least one free-flight and one transmittance query of at least one chord each (a
        # transmittance alone where nothing scatters)
        return {"bytes": case["n"] * RECORD_BYTES + env + 16 * px,
                "flops": px * case["spp"] * CHORD_FLOPS * (1 if case.get("scene") == "uniform" else 2)}
    if kind == "transmittance":
        return {"bytes": case["n"] * 44 + case["rays"] * 28, "flops": case["rays"] * CHORD_FLOPS}
    if kind == "albedo":
        return {"bytes": case["n"] * RECORD_BYTES + case["points"] * 28, "flops": case["points"] * 30}
    if kind == "emission":
        px = case["width"] * case["height"]
        return {"bytes": case["n"] * RECORD_BYTES + 16 * px, "flops": px * case["spp"] * CHORD_FLOPS}
    if kind == "train":
        px = case["width"] * case["height"] * case["views"]
        return {"bytes": case["n"] * RECORD_BYTES * 2 + 24 * px, "flops": px * case["spp"] * CHORD_FLOPS * 3}
    trace = _requests(case, 0)
    paths = sum(r.paths for r in trace)
    px = sum(r.config.image_width * r.config.image_height for r in trace)
    return {"bytes": (case["n0"] + case["n1"]) * RECORD_BYTES + 2048 * 1024 * 12 + px * 16,
            "flops": paths * CHORD_FLOPS * 2}


# ---- closed forms in 64 bits -------------------------------------------------------------------
def _whitening(gauss, sigma, scale_is_log):
    """(W (n, 3, 3), centre (n, 3), icf (n,)) in 64 bits."""
    c, q, m = gauss.mean.double(), gauss.quat_wxyz.double(), gauss.density.double() * sigma
    s = gauss.scale.double().exp() if scale_is_log else gauss.scale.double()
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).view(-1, 3, 3)
    W = R.transpose(1, 2) / s[:, :, None]
    return W, c, m * (2 * math.pi) ** -1.5 / s.prod(1) * math.sqrt(math.pi / 2)


def _hits(W, c, o, d):
    """(ray, Gaussian) index pairs whose 3-sigma chord overlaps [0, inf), for a block of rays."""
    n = W.shape[0]
    A = W.reshape(3 * n, 3).T.contiguous()
    q = (o @ A).view(-1, n, 3) - torch.einsum("nij,nj->ni", W, c)
    w = (d @ A).view(-1, n, 3)
    a2, b, c2 = (w * w).sum(2), (q * w).sum(2), (q * q).sum(2)
    h2 = 9 - (c2 - b * b / a2)
    ok = (h2 > 0) & (-b + (h2.clamp(min=0) * a2).sqrt() > 0)
    return ok.nonzero(as_tuple=True)


def _tau(W, c, icf, o, d):
    """Optical depth of each (ray, Gaussian) pair's chord over [0, inf); one row a pair."""
    q, w = torch.einsum("kij,kj->ki", W, o - c), torch.einsum("kij,kj->ki", W, d)
    a2, b = (w * w).sum(1), (q * w).sum(1)
    rw = a2.rsqrt()
    tc = -b / a2
    p = q + tc[:, None] * w
    d2 = (p * p).sum(1)
    h = (9 - d2).clamp(min=1e-300).sqrt()
    t_in, t_out = tc - h * rw, tc + h * rw
    u0 = torch.where(t_in >= 0, -h, -tc / rw)
    tau = icf * rw * torch.exp(-0.5 * d2) * (torch.erf(h / math.sqrt(2)) - torch.erf(u0 / math.sqrt(2)))
    return torch.where((d2 < 9) & (t_out - t_in.clamp(min=0) > 1e-6), tau, torch.zeros_like(tau))


def _blocks(rays, n):
    step = max(1, int(4e7 // n))
    return [(k, min(rays, k + step)) for k in range(0, rays, step)]


def _optical_depth(W, c, icf, o, d):
    out = torch.zeros(o.shape[0], dtype=torch.float64, device="cuda")
    for a, b in _blocks(o.shape[0], W.shape[0]):
        r, k = _hits(W, c, o[a:b], d[a:b])
        out[a:b].index_add_(0, r, _tau(W[k], c[k], icf[k], o[a:b][r], d[a:b][r]))
    return out


_M64 = (1 << 64) - 1


def _i64(v):
    v &= _M64
    return v - (1 << 64) if v >> 63 else v


def _shr(x, k):
    return (x >> k) & ((1 << (64 - k)) - 1)


def _pixel_rays(case, seed, camera):
    """Jittered camera rays (pixel-major, spp a pixel): PCG32 streams hashed from pixel * spp + sample."""
    W, H, spp = case["width"], case["height"], case["spp"]
    k = torch.arange(W * H * spp, device="cuda", dtype=torch.int64)
    x = k * _i64(0xbf58476d1ce4e5b9)
    x = x ^ _shr(x, 27)
    x = x * _i64(0x94d049bb133111eb)
    x = x ^ _shr(x, 31)
    inc = (x << 1) | 1
    mul = _i64(6364136223846793005)
    state = inc + (int(seed) & 0x7FFFFFFF)      # after the first step from state 0, plus the seed
    state = state * mul + inc

    def uniform(state):
        xs = _shr(_shr(state, 18) ^ state, 27) & 0xFFFFFFFF
        rot = _shr(state, 59)
        v = ((xs >> rot) | (xs << ((32 - rot) & 31))) & 0xFFFFFFFF
        return v.float().double() * 2.0 ** -32, state * mul + inc

    jx, state = uniform(state)
    jy, state = uniform(state)
    pix = k // spp
    px, py = (pix % W).double() + (jx - 0.5), (pix // W).double() + (jy - 0.5)
    eye, at, up = (torch.tensor(v, dtype=torch.float64, device="cuda") for v in (camera.eye, camera.lookat, camera.up))
    eye, at, up = (v.float().double() for v in (eye, at, up))
    focal = (eye - at).norm()
    w = (eye - at) / focal
    u = torch.linalg.cross(up, w)
    u = u / u.norm()
    v = torch.linalg.cross(w, u)
    vh = 2 * math.tan(math.radians(camera.vfov_deg) / 2) * focal
    vw = vh * W / H
    du, dv = u * vw / W, -v * vh / H
    p00 = -w * focal - (u * vw - v * vh) / 2 + (du + dv) / 2
    d = p00 + px[:, None] * du + py[:, None] * dv
    return eye.expand_as(d), d / d.norm(dim=1, keepdim=True)


def _radiance(S, C):
    """(1 - T) C / S + T for a unit environment."""
    T = torch.exp(-S)
    a = torch.where(S > 0, -torch.expm1(-S) / S.clamp(min=1e-300), torch.ones_like(S))
    return a[:, None] * C + T[:, None]


def _emission_exact(case, seed, grads):
    params, sigma = _emission_params(case, seed)
    p64 = [p.detach().double().requires_grad_(grads) for p in params]
    spp = case["spp"]
    views = case.get("views", 1)
    images, total = [], [torch.zeros_like(p) for p in p64] if grads else None
    target = _target(case, seed).double() if grads else None
    for v in range(views):
        o, d = _pixel_rays(case, seed, _camera(seed + v))
        img = []
        step = max(spp, int(4e7 // case["n"]) // spp * spp)
        for a in range(0, o.shape[0], step):
            b = min(o.shape[0], a + step)
            with torch.set_grad_enabled(grads):
                W, c, icf = _whitening(vp.Gaussians(p64[0], p64[1], p64[2], p64[3]), sigma, True)
                with torch.no_grad():
                    r, k = _hits(W, c, o[a:b], d[a:b])
                tau = _tau(W[k], c[k], icf[k], o[a:b][r], d[a:b][r])
                S = torch.zeros(b - a, dtype=torch.float64, device="cuda").index_add(0, r, tau)
                C = torch.zeros((b - a, 3), dtype=torch.float64, device="cuda").index_add(0, r, tau[:, None] * p64[4][k])
                px = _radiance(S, C).view(-1, spp, 3).mean(1)
                if grads:
                    loss = ((px - target[v].reshape(-1, 3)[a // spp:b // spp]) ** 2).sum()
                    for t, gr in zip(total, torch.autograd.grad(loss, p64)):
                        t += gr
            img.append(px.detach())
        images.append(torch.cat(img).view(case["height"], case["width"], 3))
    if grads:
        return {"images": torch.stack(images),
                **dict(zip(("mean", "log_scale", "quat", "density", "emission"), total))}
    return torch.cat([images[0], torch.ones_like(images[0][..., :1])], -1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "render" and case["scene"] == "uniform" and case["filter"] == 0.0:
        gauss, sigma = _gaussians("uniform", case["n"], seed)
        o, d = _pixel_rays(case, seed, _camera(seed))
        T = torch.exp(-_optical_depth(*_whitening(gauss, sigma, False), o, d))
        T = T.view(case["height"], case["width"], case["spp"]).mean(2)
        return torch.stack([T, T, T, torch.ones_like(T)], -1)
    if kind == "transmittance":
        gauss, sigma = _gaussians(case["scene"], case["n"], seed)
        o, d = _ray_arrays(case["rays"], seed)
        return torch.exp(-_optical_depth(*_whitening(gauss, sigma, False), o.double(), d.double()))
    if kind == "albedo":
        gauss, sigma = _gaussians(case["scene"], case["n"], seed)
        albedo = _rand(_gen(seed + 5), case["n"], 3).double()
        W, c, icf = _whitening(gauss, sigma, False)
        x = torch.from_numpy(_points(gauss, case["points"], seed)).cuda().double()
        A = W.reshape(-1, 3).T.contiguous()
        rgb = torch.zeros((x.shape[0], 3), dtype=torch.float64, device="cuda")
        for a, b in _blocks(x.shape[0], W.shape[0]):
            y = (x[a:b] @ A).view(b - a, -1, 3) - torch.einsum("nij,nj->ni", W, c)
            r2 = (y * y).sum(2)
            w = torch.where(r2 <= 9, icf * torch.exp(-0.5 * r2), torch.zeros_like(r2))
            t = w.sum(1, keepdim=True)
            rgb[a:b] = torch.where(t > 0, (w @ albedo) / t.clamp(min=1e-300), torch.zeros_like(rgb[a:b]))
        return {"rgb": rgb, "overlap": None}
    if kind == "emission":
        return _emission_exact(case, seed, False)
    if kind == "train":
        return _emission_exact(case, seed, True)
    return None  # a path-traced image has no closed form
