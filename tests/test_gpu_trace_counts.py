"""Ray-set traversal at the ray counts where the persistent kernel's use of its
warps changes (one lane per warp up to all 32, one ray more or less than the
grid's lanes), in every layout, against the plain mode (one ray per thread) and
an FP64 test of every triangle; and the records the traversal reads."""
import ctypes as C

import numpy as np
import pytest

import mcpt
from helpers import random_rays

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def scene():
    ctx = mcpt.Context(0)
    s = mcpt.generate_scene(mcpt.SCENE_BATCH_MEMBER, variant=1, seed=9, triangle_target=1500)
    tris = mcpt.host_triangles(s)
    d = mcpt.DeviceScene(tris, ctx=ctx)
    v = np.frombuffer(tris, dtype=np.uint8).reshape(len(tris), 224)[:, :36].copy().view(np.float32)
    bvhs = {l: mcpt.Bvh(ctx, d.view, layout=l) for l in (mcpt.LAYOUT_BINARY, mcpt.LAYOUT_WIDE4, mcpt.LAYOUT_WIDE4Q)}
    yield ctx, d, v, bvhs
    for b in bvhs.values():
        b.close()
    mcpt.free_scene(s)


def closest(ctx, d, bvh, rays, mode=0):
    n = rays.shape[1]
    h = torch.full((n, 4), -7, dtype=torch.int32, device="cuda")
    mcpt.check(ctx.lib.mc_trace_closest(ctx.handle, bvh.handle, C.byref(d.view), rays.data_ptr(), n, mode, h.data_ptr()))
    return h


def brute(v, rays):
    """FP64 closest t of every ray (1e30: none) over all triangles."""
    t64 = torch.from_numpy(v).cuda().double()
    r = rays.double()
    v0, e1, e2 = t64[:, 0:3], t64[:, 3:6] - t64[:, 0:3], t64[:, 6:9] - t64[:, 0:3]
    n = torch.linalg.cross(e1, e2)
    o, d = r[0:3].T, r[3:6].T
    det = -(d @ n.T)
    m = torch.linalg.cross(o, d)
    u = (m @ e2.T - d @ torch.linalg.cross(e2, v0).T) / det
    w = (d @ torch.linalg.cross(e1, v0).T - m @ e1.T) / det
    t = (o @ n.T - (v0 * n).sum(-1)) / det
    return torch.where((u >= 0) & (w >= 0) & (u + w <= 1) & (t > 1e-4), t, 1e30).min(-1).values


@pytest.mark.parametrize("n", [1, 31, 33, 4143, 4145, 151551, 151553])
def test_ray_counts(scene, n):
    ctx, d, v, bvhs = scene
    rays = torch.from_numpy(random_rays(n, -1.5, 1.5, n)).cuda()
    want = closest(ctx, d, bvhs[mcpt.LAYOUT_WIDE4], rays, mcpt.TRACE_PLAIN)
    for b in bvhs.values():
        assert torch.equal(closest(ctx, d, b, rays), want)
    occ = torch.empty(n, dtype=torch.int32, device="cuda")
    tmax = torch.full((n,), 0.75, device="cuda")
    for b in bvhs.values():
        mcpt.check(ctx.lib.mc_trace_any(ctx.handle, b.handle, C.byref(d.view), rays.data_ptr(), tmax.data_ptr(), n, 0,
                                        occ.data_ptr()))
        assert torch.equal(occ != 0, want[:, 0].view(torch.float32) < 0.75)
    k = min(n, 4096)
    t, ref = want[:k, 0].view(torch.float32).double().clamp(max=1e6), brute(v, rays[:, :k]).clamp(max=1e6)  # misses: 1e30
    # a plane distance in FP32: cancellation in (v0 - o).n over |d.n| for boxes of size about 3;
    # rays within rounding of an edge may differ altogether
    far = (t - ref).abs() > 1e-4 * ref.clamp(max=10.0)
    assert int(far.sum()) <= max(1, k // 500)


def test_exported_records_hold_the_primitives(scene):
    _, _, v, bvhs = scene
    for b in bvhs.values():
        _, prims = b.traversal_arrays()
        p = prims.cpu().numpy().reshape(-1, 48)
        ids = p.view(np.int32).reshape(-1, 12)[:, 9]
        assert sorted(ids.tolist()) == list(range(len(v)))
        assert np.array_equal(p.view(np.float32).reshape(-1, 12)[:, :9], v[ids])
