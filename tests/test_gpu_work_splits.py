"""The sizes at which kernels split their work differently. Clustering: tiles of
240 positions, one block alone up to four tiles (960). Persistent traversal: a
warp takes as many lanes as its share of the rays, 1 to 32, with 32 resident
warps per SM (4-wide trees, 128-thread blocks) or 24 (256-thread blocks); sets of
at most 8,192 closest-hit rays push children in full order."""
import ctypes as C

import numpy as np
import pytest

import mcpt
from test_gpu_build_sizes import Scene, hits

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TILE, ALONE = 240, 960


@pytest.fixture(scope="module")
def ctx():
    c = mcpt.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n", [k + d for k in (TILE, 2 * TILE, ALONE, ALONE + TILE, 148 * TILE) for d in (-1, 0, 1)])
def test_single_builds(ctx, n):
    s = Scene(ctx, n, n)
    coop = mcpt.Bvh(ctx, s.view, layout=mcpt.LAYOUT_WIDE4)
    phase = mcpt.Bvh(ctx, s.view, layout=mcpt.LAYOUT_WIDE4, phase_launches=True)
    binary = mcpt.Bvh(ctx, s.view, layout=mcpt.LAYOUT_BINARY)
    for x, y in zip(coop.traversal_arrays(), phase.traversal_arrays()):
        assert torch.equal(x, y)
    assert torch.equal(hits(ctx, s.view, coop), hits(ctx, s.view, binary))
    for b in (coop, phase, binary):
        b.close()


@pytest.mark.parametrize("total", [TILE - 1, TILE, TILE + 1, 2 * TILE, ALONE - 1, ALONE, ALONE + 1])
@pytest.mark.parametrize("scenes", [2, 7])
def test_batch_builds(ctx, total, scenes):
    """Scenes whose borders lie inside tiles, the sizes adding up to the total."""
    cut = [total * k // scenes + (k % 3 if 0 < k < scenes else 0) for k in range(scenes + 1)]
    parts = [Scene(ctx, b - a, 31 * total + a) for a, b in zip(cut, cut[1:])]
    views = [p.view for p in parts]
    trees = [mcpt.BatchBvh(ctx, views, phase_launches=p) for p in (False, True)]
    a, b = (mcpt.traversal_arrays(t.lib, t.handle) for t in trees)
    for x, y in zip(a, b):
        assert torch.equal(x, y)
    for t in trees:
        t.close()


def counts(per_sm):
    warps = torch.cuda.get_device_properties(0).multi_processor_count * per_sm
    out = []
    for k in (1, 2, 3, 8, 17, 30, 31, 32):
        out += [k * warps - 1, k * warps, k * warps + 1]
    return out + [33 * warps + 5, 8191, 8192, 8193]  # closest hits push in full order up to 8192


@pytest.mark.parametrize("layout,per_sm", [(mcpt.LAYOUT_WIDE4, 32), (mcpt.LAYOUT_WIDE4Q, 32), (mcpt.LAYOUT_BINARY, 24)])
@pytest.mark.parametrize("intersector", [mcpt.ISECT_REFERENCE, mcpt.ISECT_WATERTIGHT])
def test_lanes_per_warp(ctx, layout, per_sm, intersector):
    s = Scene(ctx, 2000, 5)
    bvh = mcpt.Bvh(ctx, s.view, layout=layout)
    if intersector == mcpt.ISECT_WATERTIGHT:
        per_sm = 24
    sizes = counts(per_sm)
    r = np.random.default_rng(3)
    most = max(sizes)
    d = r.normal(size=(3, most))
    full = np.concatenate([r.uniform(-1.2, 1.2, (3, most)), d / np.linalg.norm(d, axis=0), np.zeros((1, most))])
    full = torch.from_numpy(full.astype(np.float32)).cuda()
    tmax = torch.full((most,), 0.4, device="cuda")

    def trace(n, mode):
        rays = full[:, :n].contiguous()
        h = torch.full((n, 4), -7, dtype=torch.int32, device="cuda")
        o = torch.full((n,), -7, dtype=torch.int32, device="cuda")
        mcpt.check(ctx.lib.mc_trace_closest(ctx.handle, bvh.handle, C.byref(s.view), rays.data_ptr(), n, mode, h.data_ptr()))
        mcpt.check(ctx.lib.mc_trace_any(ctx.handle, bvh.handle, C.byref(s.view), rays.data_ptr(), tmax.data_ptr(), n, mode,
                                        o.data_ptr()))
        return h, o
    hit, occluded = trace(most, intersector | mcpt.TRACE_PLAIN)
    assert 0 < int(occluded.sum()) < most
    for n in sizes:
        h, o = trace(n, intersector)
        assert torch.equal(h, hit[:n]) and torch.equal(o, occluded[:n]), n
    bvh.close()
