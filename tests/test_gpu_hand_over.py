"""Which paths the few-paths kernel takes follows from their number and from the
bounces that remain; whatever it takes, images, random draws and ray counts
equal those of the separate launches (the plain mode): whole waves on both
sides of the limits, hand-overs with few and with many bounces left, deep waves
whose counters have gone round their ring, batches, and density grids."""
import ctypes as C

import numpy as np
import pytest

import mcpt
from test_gpu_few_paths import mixed_scene, render

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ctx():
    c = mcpt.Context(0)
    yield c
    c.close()


def same(ctx, dev, bvh, cam, w, h, spp, depth, **kw):
    a = render(ctx, dev, bvh, cam, w, h, spp, depth, persistent=True, **kw)
    b = render(ctx, dev, bvh, cam, w, h, spp, depth, persistent=False, **kw)
    assert torch.equal(a[0], b[0])
    assert a[1:] == b[1:]
    assert float(a[0].sum()) > 0
    return a


@pytest.fixture(scope="module")
def mixed(ctx):
    s, tris = mixed_scene(5, target=3000)
    d = mcpt.DeviceScene(tris, ctx=ctx)
    trees = {k: mcpt.Bvh(ctx, d.view, layout=k) for k in (mcpt.LAYOUT_BINARY, mcpt.LAYOUT_WIDE4)}
    yield s, d, trees
    for b in trees.values():
        b.close()
    mcpt.free_scene(s)


# paths at and past the limits of a whole wave: 16,384 up to depth 4, 4,096 a
# bounce up to 65,536 from depth 16 on; 65,536 in the binary layout
@pytest.mark.parametrize("w,h,depth", [(128, 128, 1), (128, 129, 1), (128, 129, 2), (128, 128, 4), (128, 129, 4),
                                       (128, 160, 5), (128, 161, 5), (256, 128, 8), (256, 129, 8), (256, 240, 15),
                                       (256, 241, 15), (256, 256, 17), (256, 257, 17)])
@pytest.mark.parametrize("layout", [mcpt.LAYOUT_BINARY, mcpt.LAYOUT_WIDE4])
def test_whole_waves(ctx, mixed, w, h, depth, layout):
    s, d, trees = mixed
    same(ctx, d, trees[layout], s.camera, w, h, 1, depth)


@pytest.mark.parametrize("depth", [2, 3, 4, 5, 7, 8, 9, 16, 33, 64])
@pytest.mark.parametrize("graph", [False, True])
def test_hand_over(ctx, mixed, depth, graph):
    """A wave of 90,000 paths leaves its last bounces to the kernel, or none where too few remain."""
    s, d, trees = mixed
    same(ctx, d, trees[mcpt.LAYOUT_WIDE4], s.camera, 300, 300, 1, depth, use_graph=graph)


@pytest.mark.parametrize("depth", [65, 100, 300])
def test_deep_hand_over(ctx, mixed, depth):
    """More paths than a whole wave holds, handed over at a read-back."""
    s, d, trees = mixed
    same(ctx, d, trees[mcpt.LAYOUT_WIDE4], s.camera, 300, 300, 1, depth)


def test_deep_hand_over_past_the_ring(ctx):
    """A closed box whose paths live on: more than 65,536 of 1.7M pass bounce
    64, so the hand-over's counters lie in a slot used before."""
    s = mcpt.generate_scene(mcpt.SCENE_CORNELL_BOXES)
    tris = mcpt.host_triangles(s)
    v = np.frombuffer(tris, dtype=np.uint8).reshape(len(tris), 224)[:, :36].copy().view(np.float32).reshape(-1, 3)
    eye = np.array([s.camera.look_from.x, s.camera.look_from.y, s.camera.look_from.z])
    lo, hi = np.minimum(v.min(0), eye) - 1.0, np.maximum(v.max(0), eye) + 1.0
    corner = lambda k: mcpt.Vec3(*[float((hi if k >> a & 1 else lo)[a]) for a in range(3)])
    inward = lambda a, side: mcpt.Vec3(*[(-1.0 if side else 1.0) if k == a else 0.0 for k in range(3)])
    box = []
    for face in ((0, 1, 3, 2), (4, 5, 7, 6), (0, 1, 5, 4), (2, 3, 7, 6), (0, 2, 6, 4), (1, 3, 7, 5)):
        for a, b, c in ((0, 1, 2), (0, 2, 3)):
            t = mcpt.Triangle.from_buffer_copy(bytes(tris[0]))
            t.v0, t.v1, t.v2 = (corner(face[k]) for k in (a, b, c))
            axis = next(x for x in range(3) if len({k >> x & 1 for k in face}) == 1)
            t.n0 = t.n1 = t.n2 = inward(axis, face[0] >> axis & 1)
            t.mat.type = mcpt.MAT_CONDUCTOR
            box.append(t)
    out = (mcpt.Triangle * (len(tris) + len(box)))(*list(tris), *box)
    for t in out:
        if t.mat.type != mcpt.MAT_EMISSIVE:
            t.mat.type, t.mat.fuzz = mcpt.MAT_CONDUCTOR, 0.3
            t.mat.albedo.type = 0
            t.mat.albedo.color_a = mcpt.Vec3(0.972, 0.972, 0.972)
    d = mcpt.DeviceScene(out, ctx=ctx)
    b = mcpt.Bvh(ctx, d.view, layout=mcpt.LAYOUT_WIDE4)
    cam = mcpt.Camera.from_buffer_copy(bytes(s.camera))
    cam.rr_cap = 1.0
    r = same(ctx, d, b, cam, 1300, 1300, 1, 300)
    extend = r[1]
    # the count is read at bounces 8, 16, .. 64, 72, and slot 0 is used again from bounce 65 on
    assert extend[62] > 72000, extend
    b.close()
    mcpt.free_scene(s)


@pytest.mark.parametrize("depths", [(3, 6, 9, 12), (64, 2, 5, 30), (100, 7, 1, 4)])
@pytest.mark.parametrize("graph", [False, True])
def test_batches_hand_over(ctx, depths, graph):
    parts = [mixed_scene(k, target=500 + 900 * k) for k in range(4)]
    devs = [mcpt.DeviceScene(t, ctx=ctx) for _, t in parts]
    batch = mcpt.BatchBvh(ctx, [d.view for d in devs])
    got = []
    for persistent in (True, False):
        accs, items = [], []
        for k, ((s, _), d) in enumerate(zip(parts, devs)):
            w = 170 + 41 * k
            c = mcpt.Camera.from_buffer_copy(bytes(s.camera))
            c.image_width, c.aspect_ratio = w, 1.0
            mcpt.camera_initialize(c)
            a = torch.zeros(w * w * 3, dtype=torch.float32, device="cuda")
            accs.append(a)
            items.append(mcpt.BatchItem(d.view, mcpt.render_params(c, w, w, 1 + (k & 1), depths[k], persistent=persistent,
                                                                   seed=k), a.data_ptr()))
        st = batch.render(items, use_graph=graph)
        got.append((accs, list(st.extend_per_depth), list(st.shadow_per_depth)))
    assert got[0][1:] == got[1][1:]
    for a, b in zip(got[0][0], got[1][0]):
        assert torch.equal(a, b)
    batch.close()
    for s, _ in parts:
        mcpt.free_scene(s)


@pytest.mark.parametrize("w,h,depth", [(400, 330, 2), (400, 330, 4), (512, 512, 8), (512, 513, 8), (1030, 1030, 8),
                                       (1030, 1030, 40), (1030, 1030, 70)])
def test_density_grids(ctx, w, h, depth):
    """132,000 to 1,060,900 paths: whole waves, hand-overs, and a deep hand-over."""
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
