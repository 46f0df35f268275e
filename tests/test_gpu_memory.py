"""GPU: the device memory that a context's pool keeps between calls (at most 2 GiB) is there for every allocation of
the process that needs it -- another context's scenes, workspaces and servers, and other allocators': the driver
takes it from the pool before an allocation fails.

The device is filled up to less than what the calls need, so that they only fit into what the pool keeps.
"""
import numpy as np
import pytest

import volprim_b200 as vp
from volprim_b200 import scenes, serving

pytestmark = pytest.mark.gpu
GIB = 1 << 30


def free_bytes():
    import torch
    return torch.cuda.mem_get_info()[0]


def fill(leave):
    """Holds device memory until at most `leave` bytes are free (blocks of at most 16 GiB, then finer ones)."""
    import torch
    held = []
    for block in (16 * GIB, GIB, GIB // 16):
        while free_bytes() > leave + block:
            held.append(torch.empty(block, dtype=torch.uint8, device="cuda"))
    return held


@pytest.fixture
def kept(vp_ctx):
    """A context whose pool keeps more than 1 GiB, nothing else cached."""
    import torch
    torch.cuda.empty_cache()
    ctx = vp.Context(0)
    rng = np.random.default_rng(1)
    n = 3_000_000
    g = vp.Gaussians(rng.uniform(-1, 1, (n, 3)).astype(np.float32), np.full((n, 3), 0.01, np.float32),
                     np.tile(np.array([1.0, 0, 0, 0], np.float32), (n, 1)), np.full(n, 1e-6, np.float32))
    before = free_bytes()
    vp.Scene(ctx, g, 1.0).close()
    ctx.synchronize()
    assert before - free_bytes() > GIB
    yield ctx
    ctx.close()
    torch.cuda.empty_cache()


@pytest.mark.parametrize("what", ["server", "render", "scene", "rays", "torch"])
def test_other_allocations_get_it(vp_ctx, kept, what):
    # everything small first: kernels loaded, workspaces in place
    g = scenes.absorption_gaussians(256, 0)
    sc = vp.Scene(vp_ctx, g, 1.0)
    env = vp.Environment(vp_ctx, constant=(1.0, 1.0, 1.0))
    cam = scenes.negz_camera()
    vp.Renderer(vp.Config(num_samples_per_pixel=1, image_width=32, image_height=32), sc, cam, env=env, ctx=vp_ctx).render()
    sc.transmittance(np.zeros((4, 3), np.float32), np.tile(np.array([0, 0, 1], np.float32), (4, 1)))
    n = 1_500_000
    rng = np.random.default_rng(2)
    big = vp.Gaussians(rng.uniform(-1, 1, (n, 3)).astype(np.float32), np.full((n, 3), 0.01, np.float32),
                       np.tile(np.array([1.0, 0, 0, 0], np.float32), (n, 1)), np.full(n, 1e-6, np.float32))
    vp.Scene(vp_ctx, scenes.absorption_gaussians(5000, 0), 1.0).close()
    o = np.zeros((30_000_000, 3), np.float32) if what == "rays" else None
    held = fill(GIB // 2)
    try:
        if what == "server":  # 2^22 slots of 264 bytes
            serving.Server(vp_ctx, path_slots=1 << 22).close()
        elif what == "render":  # 3.7M paths of some 280 bytes
            cfg = vp.Config(num_samples_per_pixel=4, image_width=1024, image_height=900, batch_spp=4)
            assert np.isfinite(vp.Renderer(cfg, sc, cam, env=env, ctx=vp_ctx).render()).all()
        elif what == "scene":  # some 600 bytes a Gaussian while building
            vp.Scene(vp_ctx, big, 1.0).close()
        elif what == "torch":
            import torch
            assert torch.empty(GIB, dtype=torch.uint8, device="cuda").numel() == GIB
        else:  # 28 bytes a ray
            assert sc.transmittance(o, np.broadcast_to(np.array([0, 0, 1], np.float32), o.shape)).shape == (30_000_000,)
    finally:
        del held
        import torch
        torch.cuda.empty_cache()
        env.close()
        sc.close()


def test_a_build_without_room_for_the_8_wide_tree(vp_ctx):
    """A device with room for everything else builds the scene without it, and queries give the same: the free memory
    goes down in steps of 32 MiB from where all of it fits until the rest does not (the tree's scratch is some 80 bytes
    a Gaussian more than what the build frees before it)."""
    import torch
    from test_gpu_few_paths import has_8_wide_tree
    n = 2_000_000
    rng = np.random.default_rng(3)
    g = vp.Gaussians(rng.uniform(-1, 1, (n, 3)).astype(np.float32), np.full((n, 3), 0.01, np.float32),
                     np.tile(np.array([1.0, 0, 0, 0], np.float32), (n, 1)), np.full(n, 1e-5, np.float32))
    how = dict(wide_builder="lbvh", binary_builder="lbvh", collapse="greedy")
    o = np.tile(np.array([0.1, 0.2, -3.0], np.float32), (1000, 1))
    d = np.concatenate([rng.uniform(-0.3, 0.3, (1000, 2)), np.ones((1000, 1))], 1)
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    torch.cuda.empty_cache()
    ctx = vp.Context(0)
    sc = vp.Scene(ctx, g, 1.0, **how)
    assert has_8_wide_tree(sc.info())
    want = sc.transmittance(o, d)
    sc.close()
    ctx.close()
    held = fill(GIB // 4)  # what other contexts' pools still keep goes first
    try:
        torch.empty(2 * GIB, dtype=torch.uint8, device="cuda")
    except torch.OutOfMemoryError:
        pass
    held = None
    torch.cuda.empty_cache()
    without = 0
    for leave in range(1280, 800, -32):
        ctx = vp.Context(0)
        held = fill(leave << 20)
        try:
            sc = vp.Scene(ctx, g, 1.0, **how)
        except vp.VpError as e:
            assert "OUT_OF_MEMORY" in str(e)
            break
        else:
            if not has_8_wide_tree(sc.info()):
                without += 1
                del held
                torch.cuda.empty_cache()
                assert np.abs(sc.transmittance(o, d) - want).max() <= 1e-7
            sc.close()
        finally:
            held = None
            torch.cuda.empty_cache()
            ctx.close()
    assert without > 0
