"""The octant form of the 4-wide nodes against the 128-byte nodes and the binary
tree: rays of every direction octant, with zero components of either sign, on
both sides of the size rule, and shared waves whose trees are of both kinds."""
import ctypes as C
import itertools

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


def scene(target, variant=4):
    s = mcpt.generate_scene(mcpt.SCENE_BATCH_MEMBER, variant=variant, seed=2, triangle_target=target)
    return s, mcpt.DeviceScene(mcpt.host_triangles(s))


def octant_rays(per):
    """Rays of all sign patterns, some components exactly +0 or -0."""
    r = np.random.default_rng(per)
    out = []
    for sign in itertools.product([1, -1], repeat=3):
        for zero in itertools.product([0, 1], repeat=3):
            if all(zero):
                continue
            d = r.uniform(0.1, 1, (3, per)) * np.where(zero, 0.0, 1.0)[:, None]
            d = np.copysign(d / np.linalg.norm(d, axis=0), np.array(sign)[:, None])
            out.append(np.concatenate([r.uniform(-1, 1, (3, per)), d, r.uniform(0, 1, (1, per))]))
    return torch.from_numpy(np.concatenate(out, 1).astype(np.float32)).cuda()


@pytest.mark.parametrize("target", [2, 700, 40000, 900000])
def test_octants(ctx, target):
    s, d = scene(target)
    rays = octant_rays(37)
    n = rays.shape[1]
    got = []
    for layout in (mcpt.LAYOUT_BINARY, mcpt.LAYOUT_WIDE4, mcpt.LAYOUT_WIDE4Q):
        for builder in (mcpt.BUILDER_CLUSTERED, mcpt.BUILDER_LBVH):
            b = mcpt.Bvh(ctx, d.view, layout=layout, builder=builder)
            for mode in (0, mcpt.TRACE_PLAIN):
                h = torch.empty(n, 4, dtype=torch.int32, device="cuda")
                mcpt.check(ctx.lib.mc_trace_closest(ctx.handle, b.handle, C.byref(d.view), rays.data_ptr(), n, mode,
                                                    h.data_ptr()))
                got.append(h)
            b.close()
    assert int((got[0][:, 0].view(torch.float32) < 1e29).sum()) > n // 50
    for h in got[1:]:
        assert torch.equal(h, got[0])
    mcpt.free_scene(s)


def test_shared_waves_of_both_forms(ctx):
    """A tree with octant nodes beside one above their size limit."""
    scenes = [scene(3000, 1), scene(900000, 2)]
    want = []
    for s, d in scenes:
        cam = mcpt.Camera.from_buffer_copy(bytes(s.camera))
        cam.image_width, cam.aspect_ratio = 48, 1.0
        mcpt.camera_initialize(cam)
        p = mcpt.render_params(cam, 48, 48, 3, 8, persistent=True, rng=mcpt.RNG_PHILOX, seed=5)
        bvh = mcpt.Bvh(ctx, d.view, layout=mcpt.LAYOUT_WIDE4)
        ref = torch.zeros(48 * 48 * 3, dtype=torch.float32, device="cuda")
        st = mcpt.RenderStats()
        mcpt.check(ctx.lib.mc_render_wavefront(ctx.handle, bvh.handle, C.byref(d.view), C.byref(p), ref.data_ptr(),
                                               C.byref(st)))
        want.append((p, ref.cpu().numpy()))
        bvh.close()
    for order in ((0, 1), (1, 0)):
        srv = mcpt.Server(ctx, samples_per_step=1)
        rids = {k: srv.submit(srv.add_scene(scenes[k][1]), want[k][0]) for k in order}
        for _ in range(100):
            if srv.step() == 0 and srv.stats().pending == 0:
                break
        for k, rid in rids.items():
            assert np.array_equal(srv.read(rid, 48, 48), want[k][1])
        srv.close()
    for s, _ in scenes:
        mcpt.free_scene(s)
