"""How short a traversal stack (stack_entries) a render accepts. A ray pushes
the children of a 4-wide node farthest first, and an occlusion ray that finds
its occluder in a node needs no room for the node's other children; the least
stack of a call follows from that order and is part of what the call accepts.
Launches whose stack holds any ray push in another order; the image is the same.

The numbers are those of the renderer before it had launches of that kind."""
import ctypes as C

import pytest

import mcpt

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

STACK_OVERFLOW = 4
SMALL, LARGE = (24, 16, 1, 3), (128, 128, 2, 8)
CALLS = [(layout, rng, size) for layout in (mcpt.LAYOUT_WIDE4, mcpt.LAYOUT_WIDE4Q)
         for rng in (mcpt.RNG_XORWOW, mcpt.RNG_PHILOX) for size in (SMALL, LARGE)]
# scene seed, triangle target, least stack_entries of each call of CALLS
LEAST = [
    (0, 5000, [9, 13, 8, 13, 9, 13, 8, 13]),
    (0, 40000, [10, 14, 11, 16, 11, 14, 11, 16]),
    (1, 40000, [12, 14, 10, 14, 12, 14, 11, 15]),
    (2, 40000, [11, 17, 12, 13, 12, 17, 13, 14]),
    (8, 40000, [10, 14, 10, 13, 10, 14, 10, 13]),
    (10, 5000, [10, 12, 10, 12, 10, 13, 10, 13]),
    (11, 5000, [10, 12, 9, 13, 11, 12, 10, 14])]


@pytest.fixture(scope="module")
def ctx():
    c = mcpt.Context(0)
    yield c
    c.close()


def render(ctx, s, d, b, rng, size, stack, **kw):
    w, h, spp, depth = size
    c = mcpt.Camera.from_buffer_copy(bytes(s.camera))
    c.image_width, c.image_height, c.aspect_ratio = w, h, w / float(h)
    mcpt.camera_initialize(c)
    p = mcpt.render_params(c, w, h, spp, depth, seed=77, rng=rng, stack_entries=stack, **kw)
    if rng == mcpt.RNG_XORWOW:
        mcpt.check(ctx.lib.mc_rng_reset(ctx.handle, w, h, 77))
    acc = torch.zeros(w * h * 3, dtype=torch.float32, device="cuda")
    st = ctx.lib.mc_render_wavefront(ctx.handle, b.handle, C.byref(d.view), C.byref(p), acc.data_ptr(), None)
    return st, acc


@pytest.mark.parametrize("seed,target,least", LEAST)
def test_least_stack(ctx, seed, target, least):
    s = mcpt.generate_scene(mcpt.SCENE_BATCH_MEMBER, variant=seed, seed=seed + 1, triangle_target=target)
    d = mcpt.DeviceScene(mcpt.host_triangles(s), ctx=ctx)
    trees = {k: mcpt.Bvh(ctx, d.view, layout=k) for k in (mcpt.LAYOUT_WIDE4, mcpt.LAYOUT_WIDE4Q)}
    for (layout, rng, size), n in zip(CALLS, least):
        for kw in ({}, dict(persistent=False), dict(trace_threads=128)):
            b = trees[layout]
            st, image = render(ctx, s, d, b, rng, size, 0, **kw)
            assert st == 0
            st, short = render(ctx, s, d, b, rng, size, n, **kw)
            assert st == 0 and torch.equal(image, short), (layout, rng, size, kw)
            assert render(ctx, s, d, b, rng, size, n - 1, **kw)[0] == STACK_OVERFLOW, (layout, rng, size, kw)
    for b in trees.values():
        b.close()
    mcpt.free_scene(s)
