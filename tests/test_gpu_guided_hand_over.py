"""Guided renders hand their last paths to the few-paths kernel only past the
guided bounces: image, random draws, ray counts and trained weights equal those
of the separate launches (the plain mode, which never hands over), whatever the
guided depth, below and above the depth at which a wave's counters are a ring."""
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


@pytest.fixture(scope="module", params=[mcpt.SCENE_CORNELL_BOXES, mcpt.SCENE_GUIDING_ROOM])
def scene(request, ctx):
    s = mcpt.generate_scene(request.param)
    tris = mcpt.host_triangles(s)
    d = mcpt.DeviceScene(tris, ctx=ctx)
    b = mcpt.Bvh(ctx, d.view, layout=mcpt.LAYOUT_WIDE4)
    v = np.frombuffer(tris, dtype=np.uint8).reshape(len(tris), 224)[:, :36].copy().view(np.float32).reshape(-1, 3)
    yield s, d, b, v.min(0).tolist(), v.max(0).tolist()
    b.close()
    mcpt.free_scene(s)


def guided(ctx, scene, w, spp, depth, persistent, train, **cfg):
    s, d, b, lo, hi = scene
    cam = mcpt.Camera.from_buffer_copy(bytes(s.camera))
    cam.image_width, cam.aspect_ratio = w, 1.0
    mcpt.camera_initialize(cam)
    guide = mcpt.Guide(ctx, lo, hi, seed=3, **cfg)
    p = mcpt.render_params(cam, w, w, spp, depth, persistent=persistent, seed=77)
    acc = torch.zeros(w * w * 3, dtype=torch.float32, device="cuda")
    st = mcpt.RenderStats()
    mcpt.check(ctx.lib.mc_render_guided(ctx.handle, b.handle, C.byref(d.view), C.byref(p), guide.handle, train,
                                        acc.data_ptr(), C.byref(st)))
    assert st.error_flags == 0
    weights = guide.get_params()
    guide.close()
    return acc, list(st.extend_per_depth), list(st.shadow_per_depth), weights


@pytest.mark.parametrize("w,spp,depth,guided_depth", [
    (64, 1, 100, 16),      # deep, guided past the first read-back of the path count
    (64, 1, 100, 1024),    # deep, every bounce guided
    (300, 1, 100, 9),      # deep, more paths than one launch takes at the start
    (64, 1, 100, 4),       # deep, unguided from the first read-back on
    (300, 1, 40, 16),      # not deep: handed over at the end of the wave
    (300, 1, 40, 1024),
    (300, 1, 40, 1),
    (160, 2, 8, 2)])
def test_hand_over_keeps_the_guided_bounces(ctx, scene, w, spp, depth, guided_depth):
    a = guided(ctx, scene, w, spp, depth, True, 0, guided_depth=guided_depth)
    b = guided(ctx, scene, w, spp, depth, False, 0, guided_depth=guided_depth)
    assert torch.equal(a[0], b[0])
    assert a[1:3] == b[1:3]
    assert float(a[0].sum()) > 0


@pytest.mark.parametrize("depth,guided_depth,vertices", [(100, 16, 4), (40, 2, 1), (40, 4, 4)])
def test_hand_over_keeps_the_training(ctx, scene, depth, guided_depth, vertices):
    kw = dict(guided_depth=guided_depth, train_vertices=vertices, learning_rate=3e-3)
    a = guided(ctx, scene, 160, 2, depth, True, 1, **kw)
    b = guided(ctx, scene, 160, 2, depth, False, 1, **kw)
    assert torch.equal(a[0], b[0])
    assert a[1:3] == b[1:3]
    assert np.array_equal(np.asarray(a[3]), np.asarray(b[3]))
