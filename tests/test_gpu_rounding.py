"""Images do not depend on which kernel shades a path or traces a ray: the
few-paths kernel equals the separate launches in every layout, and the XORWOW and
Philox kernels round as they always have. The digests are those of the
accumulation buffers before the few-paths kernel existed, when every expression
was left to one kernel's compilation."""
import ctypes as C
import hashlib

import numpy as np
import pytest

import mcpt
from test_gpu_few_paths import mixed_scene, render, same

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ctx():
    c = mcpt.Context(0)
    yield c
    c.close()


def cloud(ctx):
    dens, org = mcpt.fog_sphere(60.0, 6.0)
    g, hd = mcpt.volume_grid_create(ctx, dens * 0.02, tuple(np.asarray(org, np.float32) + np.float32([0, 100, -40])), 6.0)
    s = mcpt.SceneHost()
    mcpt.check(ctx.lib.mc_scene_cloud(g, C.byref(hd), 1, C.byref(s)))
    return s, g


def scene(ctx, name):
    """(scene, device scene, what to destroy afterwards)"""
    grid, env = None, None
    if name.startswith("mixed"):
        k = int(name[5:])
        s, tris = mixed_scene(k, target=(300, 2000, 30000)[k])
        env = np.random.default_rng(1).uniform(0, 2, (16, 32, 4)).astype(np.float32) if k else None
    elif name == "cloud":
        s, grid = cloud(ctx)
        tris = mcpt.host_triangles(s)
    else:
        s = {"boxes": lambda: mcpt.generate_scene(mcpt.SCENE_CORNELL_BOXES),
             "spheres": lambda: mcpt.generate_scene(mcpt.SCENE_CORNELL_SPHERES, seed=4),
             "icospheres": lambda: mcpt.generate_scene(mcpt.SCENE_DISPLACED_ICOSPHERES, variant=3, seed=2)}[name]()
        tris = mcpt.host_triangles(s)
        env = mcpt.host_env(s) if name == "icospheres" else None
    spheres = None if name.startswith("mixed") else mcpt.host_spheres(s)
    return s, mcpt.DeviceScene(tris, spheres=spheres, env_rgba=env, ctx=ctx), grid


SCENES = ["mixed0", "mixed1", "mixed2", "boxes", "spheres", "icospheres", "cloud"]
LAYOUTS = [mcpt.LAYOUT_BINARY, mcpt.LAYOUT_WIDE4, mcpt.LAYOUT_WIDE4Q]


@pytest.mark.parametrize("name", SCENES)
@pytest.mark.parametrize("layout", LAYOUTS)
def test_few_paths_in_every_layout(ctx, name, layout):
    s, d, grid = scene(ctx, name)
    b = mcpt.Bvh(ctx, d.view, layout=layout)
    same(ctx, d, b, s.camera, 120, 100, 1, 20)
    same(ctx, d, b, s.camera, 300, 300, 1, 9)
    b.close()
    mcpt.free_scene(s)
    if grid:
        mcpt.volume_grid_destroy(grid)


@pytest.mark.parametrize("name,size,kw,digest", [
    ("mixed0", (40, 30, 3, 8), dict(rng=mcpt.RNG_XORWOW), "78b52fd261b9"),
    ("mixed1", (200, 150, 2, 20), dict(rng=mcpt.RNG_XORWOW), "7643424a24ac"),
    ("mixed1", (200, 150, 2, 20), dict(rng=mcpt.RNG_XORWOW, env_sampling=1), "60a04e684fdc"),
    ("mixed2", (200, 150, 2, 20), dict(rng=mcpt.RNG_XORWOW), "3c6ea4681d4e"),
    ("boxes", (200, 150, 2, 20), dict(rng=mcpt.RNG_XORWOW), "677a2d4e55f3"),
    ("spheres", (200, 150, 2, 20), dict(rng=mcpt.RNG_XORWOW), "4c5847a26876"),
    ("icospheres", (200, 150, 2, 20), dict(rng=mcpt.RNG_XORWOW), "efe13666b0d7"),
    ("cloud", (333, 180, 2, 40), dict(rng=mcpt.RNG_XORWOW), "5f2198b58a91"),
    ("mixed2", (200, 150, 2, 20), dict(), "42beb0aeca30"),
    ("mixed1", (200, 150, 2, 20), dict(intersector=1), "e9949411ddcf"),
    ("mixed1", (200, 150, 2, 20), dict(env_sampling=1), "d3fa7f73ea16"),
    ("spheres", (200, 150, 2, 20), dict(), "82e02a8e1abc"),
    ("cloud", (333, 180, 2, 40), dict(), "106785cc6983")])
def test_images_keep_their_bits(ctx, name, size, kw, digest):
    s, d, grid = scene(ctx, name)
    for layout in LAYOUTS:
        b = mcpt.Bvh(ctx, d.view, layout=layout)
        for persistent in (True, False):
            image = render(ctx, d, b, s.camera, *size, persistent, **kw)[0]
            assert hashlib.sha1(image.cpu().numpy().tobytes()).hexdigest()[:12] == digest, (layout, persistent)
        b.close()
    mcpt.free_scene(s)
    if grid:
        mcpt.volume_grid_destroy(grid)


@pytest.mark.parametrize("name,stack", [("spheres", 14), ("mixed1", 20), ("mixed2", 20), ("boxes", 8)])
@pytest.mark.parametrize("layout", [mcpt.LAYOUT_WIDE4, mcpt.LAYOUT_WIDE4Q])
def test_short_stacks_keep_the_image(ctx, name, stack, layout):
    """Launches that push in full order (a stack below 3 entries per level)."""
    s, d, _ = scene(ctx, name)
    b = mcpt.Bvh(ctx, d.view, layout=layout)
    assert stack < 3 * b.info().wide_levels
    for rng in (mcpt.RNG_PHILOX, mcpt.RNG_XORWOW):
        for persistent in (True, False):
            want = render(ctx, d, b, s.camera, 150, 120, 1, 20, persistent, rng=rng)
            got = render(ctx, d, b, s.camera, 150, 120, 1, 20, persistent, rng=rng, stack_entries=stack)
            assert torch.equal(want[0], got[0]) and want[1:] == got[1:]
    b.close()
    mcpt.free_scene(s)
