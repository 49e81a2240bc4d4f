"""Waves of few paths run as one launch that carries each path to its end; the
image, the random draws and the ray counts equal those of the wave's separate
launches (which the plain mode always uses), for every material, light, texture
and layout, for one scene and for batches, and for deep renders that hand their
last paths over."""
import ctypes as C

import numpy as np
import pytest

import mcpt

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ctx():
    c = mcpt.Context(0)
    yield c
    c.close()


def mixed_scene(seed, base=mcpt.SCENE_BATCH_MEMBER, target=1200):
    """A generated scene with every material type, tilted lights, checkers, smooth normals and texture coordinates."""
    s = mcpt.generate_scene(base, variant=seed & 1, seed=seed + 3, triangle_target=target)
    r = np.random.default_rng(seed)
    tris = mcpt.host_triangles(s)
    for i, t in enumerate(tris):
        m = t.mat
        k = r.integers(0, 16)
        if k < 3:
            m.type, m.fuzz = mcpt.MAT_CONDUCTOR, float(r.uniform(0, 0.4))
        elif k < 5:
            m.type, m.refraction_index = mcpt.MAT_DIELECTRIC, 1.5
        elif k == 5:
            m.type, m.emitted = mcpt.MAT_EMISSIVE, mcpt.Vec3(*[float(x) for x in r.uniform(0.2, 3, 3)])
        elif k < 9:
            m.albedo.type, m.albedo.scale = mcpt.TEX_CHECKER, 7.0
            m.albedo.color_b = mcpt.Vec3(*[float(x) for x in r.uniform(0.1, 0.9, 3)])
        if k & 1:
            v = [np.array([p.x, p.y, p.z]) for p in (t.v0, t.v1, t.v2)]
            n = np.cross(v[1] - v[0], v[2] - v[0])
            n = n / max(np.linalg.norm(n), 1e-20)
            for f in ("n0", "n1", "n2"):
                q = n + r.normal(size=3) * 0.2
                setattr(t, f, mcpt.Vec3(*[float(x) for x in q / np.linalg.norm(q)]))
            t.uv0, t.uv1, t.uv2 = mcpt.Vec2(0, 0), mcpt.Vec2(1, 0.25), mcpt.Vec2(0.5, 1)
    return s, tris


def render(ctx, dev, bvh, cam, w, h, spp, depth, persistent, **kw):
    c = mcpt.Camera.from_buffer_copy(bytes(cam))
    c.image_width, c.image_height, c.aspect_ratio = w, h, w / float(h)
    mcpt.camera_initialize(c)
    p = mcpt.render_params(c, w, h, spp, depth, persistent=persistent, seed=77, **kw)
    if kw.get("rng") == mcpt.RNG_XORWOW:
        mcpt.check(ctx.lib.mc_rng_reset(ctx.handle, w, h, 77))
    acc = torch.zeros(w * h * 3, dtype=torch.float32, device="cuda")
    st = mcpt.RenderStats()
    mcpt.check(ctx.lib.mc_render_wavefront(ctx.handle, bvh.handle, C.byref(dev.view), C.byref(p), acc.data_ptr(), C.byref(st)))
    return acc, list(st.extend_per_depth), list(st.shadow_per_depth), st.extend_rays, st.shadow_rays


def same(ctx, dev, bvh, cam, *a, **kw):
    few = render(ctx, dev, bvh, cam, *a, persistent=True, **kw)
    wave = render(ctx, dev, bvh, cam, *a, persistent=False, **kw)
    assert torch.equal(few[0], wave[0])
    assert few[1:] == wave[1:]
    assert a[0] * a[1] < 64 or float(few[0].sum()) > 0


@pytest.mark.parametrize("w,h,spp,depth,layout,rng,sky", [
    (1, 1, 1, 8, mcpt.LAYOUT_WIDE4, mcpt.RNG_PHILOX, False),
    (65, 63, 1, 8, mcpt.LAYOUT_WIDE4, mcpt.RNG_PHILOX, True),
    (127, 33, 3, 20, mcpt.LAYOUT_BINARY, mcpt.RNG_PHILOX, False),
    (128, 128, 4, 64, mcpt.LAYOUT_WIDE4Q, mcpt.RNG_PHILOX, True),   # exactly the largest one-launch wave
    (128, 129, 4, 6, mcpt.LAYOUT_WIDE4, mcpt.RNG_PHILOX, False),    # just above it
    (300, 301, 1, 40, mcpt.LAYOUT_WIDE4, mcpt.RNG_PHILOX, True),    # hands its last bounces over
    (90, 70, 2, 12, mcpt.LAYOUT_WIDE4, mcpt.RNG_XORWOW, True),
    (90, 70, 2, 1, mcpt.LAYOUT_WIDE4, mcpt.RNG_PHILOX, True)])
def test_mixed_materials(ctx, w, h, spp, depth, layout, rng, sky):
    s, tris = mixed_scene(5 + depth)
    env = None
    if sky:
        env = np.random.default_rng(1).uniform(0, 2, (16, 32, 4)).astype(np.float32)
    d = mcpt.DeviceScene(tris, env_rgba=env, ctx=ctx)
    b = mcpt.Bvh(ctx, d.view, layout=layout)
    same(ctx, d, b, s.camera, w, h, spp, depth, rng=rng)
    b.close()
    mcpt.free_scene(s)


@pytest.mark.parametrize("rng", [mcpt.RNG_PHILOX, mcpt.RNG_XORWOW])
def test_spheres_and_media(ctx, rng):
    s = mcpt.generate_scene(mcpt.SCENE_CORNELL_SPHERES, seed=4)
    d = mcpt.DeviceScene(mcpt.host_triangles(s), spheres=mcpt.host_spheres(s), ctx=ctx)
    b = mcpt.Bvh(ctx, d.view, layout=mcpt.LAYOUT_WIDE4)
    same(ctx, d, b, s.camera, 120, 100, 3, 20, rng=rng)
    same(ctx, d, b, s.camera, 60, 50, 2, 300, rng=rng)
    b.close()
    mcpt.free_scene(s)


@pytest.mark.parametrize("w,h,depth", [(61, 33, 8), (61, 33, 200), (400, 330, 200)])
def test_density_grids(ctx, w, h, depth):
    dens, org = mcpt.fog_sphere(60.0, 6.0)
    g, hd = mcpt.volume_grid_create(ctx, dens * 0.02, tuple(np.asarray(org, np.float32) + np.float32([0, 100, -40])), 6.0)
    s = mcpt.SceneHost()
    mcpt.check(ctx.lib.mc_scene_cloud(g, C.byref(hd), 1, C.byref(s)))
    d = mcpt.DeviceScene(mcpt.host_triangles(s), spheres=mcpt.host_spheres(s), ctx=ctx)
    b = mcpt.Bvh(ctx, d.view, layout=mcpt.LAYOUT_WIDE4)
    same(ctx, d, b, s.camera, w, h, 1, depth)
    b.close()
    mcpt.free_scene(s)
    mcpt.volume_grid_destroy(g)


def test_batches(ctx):
    parts = [mixed_scene(k, target=400 + 300 * k) for k in range(5)]
    devs = [mcpt.DeviceScene(t, ctx=ctx) for _, t in parts]
    batch = mcpt.BatchBvh(ctx, [d.view for d in devs])
    got = []
    for persistent in (True, False):
        accs, items = [], []
        for k, ((s, _), d) in enumerate(zip(parts, devs)):
            w = 20 + 13 * k
            c = mcpt.Camera.from_buffer_copy(bytes(s.camera))
            c.image_width, c.aspect_ratio = w, 1.0
            mcpt.camera_initialize(c)
            a = torch.zeros(w * w * 3, dtype=torch.float32, device="cuda")
            accs.append(a)
            items.append(mcpt.BatchItem(d.view, mcpt.render_params(c, w, w, 2, 2 + 3 * k, persistent=persistent, seed=k),
                                        a.data_ptr()))
        for graph in (False, True):
            st = batch.render(items, use_graph=graph)
        got.append((accs, st.extend_rays, st.shadow_rays))
    assert got[0][1:] == got[1][1:]
    for a, b in zip(got[0][0], got[1][0]):
        assert torch.equal(a, b)
    batch.close()
    for s, _ in parts:
        mcpt.free_scene(s)


def test_stack_limit_is_reported(ctx):
    s, tris = mixed_scene(2, target=3000)
    d = mcpt.DeviceScene(tris, ctx=ctx)
    b = mcpt.Bvh(ctx, d.view, layout=mcpt.LAYOUT_WIDE4)
    with pytest.raises(mcpt.McError) as e:
        render(ctx, d, b, s.camera, 64, 64, 1, 8, True, stack_entries=1)
    assert e.value.status == 4
    b.close()
    mcpt.free_scene(s)
