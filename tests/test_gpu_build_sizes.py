"""Builds at the sizes where the cooperative clustering and collapse change how
they divide their work (tiles of 240, the rounds one block runs alone, blocks
with several scenes): the same tree, byte for byte, as the launch-per-phase
loops, and the same scene bounds and hits as a build that also refits the LBVH."""
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


def triangles(n, seed):
    r = np.random.default_rng(seed)
    v = np.zeros((n, 56), np.float32)
    c = r.uniform(-1, 1, (n, 1, 3))
    size = r.choice([0.01, 0.05, 1.5], (n, 1, 1), p=[0.7, 0.29, 0.01])  # a few large ones: many small late rounds
    v[:, :9] = (c + r.uniform(-1, 1, (n, 3, 3)) * size).reshape(n, 9)
    return torch.from_numpy(v).cuda()


class Scene:
    def __init__(self, ctx, n, seed, full=None):
        full = triangles(n, seed) if full is None else full
        self.hot = torch.empty(n * 36, dtype=torch.uint8, device="cuda")
        self.cold = torch.empty(n * 192, dtype=torch.uint8, device="cuda")
        self.light = torch.zeros(64, dtype=torch.uint8, device="cuda")
        mcpt.check(ctx.lib.mc_scene_ingest(ctx.handle, full.data_ptr(), n, None, 0, self.hot.data_ptr(), self.cold.data_ptr(),
                                           None, None, None))
        v = mcpt.SceneView()
        v.tri_hot, v.tri_cold, v.triangle_count, v.lights = self.hot.data_ptr(), self.cold.data_ptr(), n, self.light.data_ptr()
        self.view, self.n = v, n


def hits(ctx, view, bvh, n=2000):
    r = np.random.default_rng(7)
    rays = np.zeros((7, n), np.float32)
    rays[0:3] = r.uniform(-1.2, 1.2, (3, n))
    d = r.normal(size=(3, n))
    rays[3:6] = d / np.linalg.norm(d, axis=0)
    rays = torch.from_numpy(rays).cuda()
    h = torch.empty(n, 4, dtype=torch.int32, device="cuda")
    mcpt.check(ctx.lib.mc_trace_closest(ctx.handle, bvh.handle, C.byref(view), rays.data_ptr(), n, 0, h.data_ptr()))
    return h


@pytest.mark.parametrize("n", [1, 2, 3, 255, 256, 257, 1023, 1024, 1025, 4099, 75777, 303105, 700001])
@pytest.mark.parametrize("builder", [mcpt.BUILDER_CLUSTERED, mcpt.BUILDER_LBVH])
def test_single(ctx, n, builder):
    s = Scene(ctx, n, n)
    coop = mcpt.Bvh(ctx, s.view, layout=mcpt.LAYOUT_WIDE4, builder=builder)
    phase = mcpt.Bvh(ctx, s.view, layout=mcpt.LAYOUT_WIDE4, builder=builder, phase_launches=True)
    refit = mcpt.Bvh(ctx, s.view, layout=mcpt.LAYOUT_WIDE4, builder=builder, keep_reference_nodes=True)
    binary = mcpt.Bvh(ctx, s.view, layout=mcpt.LAYOUT_BINARY)
    a, b, c = (x.traversal_arrays() for x in (coop, phase, refit))
    for x, y, z in zip(a, b, c):
        assert torch.equal(x, y) and torch.equal(x, z)
    i = [x.info() for x in (coop, phase, refit, binary)]
    box = [(q.scene_bounds.lo.x, q.scene_bounds.lo.y, q.scene_bounds.lo.z, q.scene_bounds.hi.x, q.scene_bounds.hi.y,
            q.scene_bounds.hi.z) for q in i]
    assert box[0] == box[1] == box[2] == box[3]
    want = hits(ctx, s.view, binary)
    for x in (coop, phase, refit):
        assert torch.equal(hits(ctx, s.view, x), want)
        x.close()
    binary.close()


def level_sizes(nodes):
    """Wide nodes per level of a tree, from its 128-byte nodes."""
    refs = nodes.cpu().numpy().view(np.int32).reshape(-1, 32)[:, 24:28]
    front, sizes = np.array([0]), []
    while len(front):
        sizes.append(len(front))
        children = refs[front].ravel()
        front = children[(children >= 0) & (children < len(refs))]
    return sizes


@pytest.mark.parametrize("chain", [21, 24, 27])
def test_frontier_that_grows_again(ctx, chain):
    """A wide level of many nodes, then a few levels of a chain, then many again:
    the collapse goes from all blocks to one and back."""
    dense = far = 30000
    r = np.random.default_rng(dense)
    c = np.concatenate([r.uniform(-0.01, 0.01, (dense, 1, 3)), np.zeros((chain, 1, 3)),
                        r.uniform(-2e6, 2e6, (far, 1, 3)) + [[[2e7, 7e5, 7e5]]]])
    size = np.concatenate([np.full(dense, 1e-3), 0.02 * 1.5 ** np.arange(chain), np.full(far, 100.0)])[:, None, None]
    shape = r.uniform(-1, 1, (len(c), 3, 3))
    shape[dense:dense + chain] = [[-1, -1, -1], [1, -1, 1], [0, 1, 0]]
    full = np.zeros((len(c), 56), np.float32)
    full[:, :9] = (c + shape * size).reshape(len(c), 9)
    s = Scene(ctx, len(c), 0, torch.from_numpy(full).cuda())
    phase = mcpt.Bvh(ctx, s.view, layout=mcpt.LAYOUT_WIDE4, phase_launches=True)
    want = phase.traversal_arrays()
    sizes = level_sizes(want[0])
    big = [k for k, n in enumerate(sizes) if n > 1024]
    assert any(n <= 1024 for n in sizes[big[0]:big[-1]]), sizes
    coop = mcpt.Bvh(ctx, s.view, layout=mcpt.LAYOUT_WIDE4)
    for x, y in zip(coop.traversal_arrays(), want):
        assert torch.equal(x, y)
    coop.close()
    phase.close()


@pytest.mark.parametrize("sizes", [(2, 2), (300, 2, 5, 1021, 7), tuple([40] * 60), (2000, 3, 90000, 511)])
def test_batch(ctx, sizes):
    scenes = [Scene(ctx, n, 100 + k) for k, n in enumerate(sizes)]
    views = [s.view for s in scenes]
    a = mcpt.BatchBvh(ctx, views)
    b = mcpt.BatchBvh(ctx, views, phase_launches=True)
    for x, y in zip(mcpt.traversal_arrays(ctx.lib, a.handle), mcpt.traversal_arrays(ctx.lib, b.handle)):
        assert torch.equal(x, y)
    a.close()
    b.close()


def test_morton_bounds_over_mixed_blocks(ctx):
    """Scene bounds of blocks that hold one scene, and their Morton codes."""
    s = Scene(ctx, 70001, 3)
    codes = torch.empty(s.n, dtype=torch.int32, device="cuda")
    box = mcpt.AABB()
    mcpt.check(ctx.lib.mc_morton_codes(ctx.handle, C.byref(s.view), codes.data_ptr(), C.byref(box)))
    v = s.hot.view(torch.float32).reshape(-1, 3)
    eps = torch.tensor(1e-3, device="cuda")
    assert [box.lo.x, box.lo.y, box.lo.z] == (v.min(0).values - eps).tolist()
    assert [box.hi.x, box.hi.y, box.hi.z] == (v.max(0).values + eps).tolist()
