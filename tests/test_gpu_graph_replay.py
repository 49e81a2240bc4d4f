"""A context replays its captured wave only for a call that would capture the
same one: after a change of the stack, the queue, the block size, the
environment sampling or the trees of a batch, the graph renders what the plain
launches of the same call render, and refuses what they refuse."""
import ctypes as C

import numpy as np
import pytest

import mcpt

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

STACK_OVERFLOW, QUEUE_OVERFLOW = 4, 5


@pytest.fixture
def ctx():
    c = mcpt.Context(0)
    yield c
    c.close()


def member(ctx, target, variant=0, env=None):
    s = mcpt.generate_scene(mcpt.SCENE_BATCH_MEMBER, variant=variant, seed=3, triangle_target=target)
    d = mcpt.DeviceScene(mcpt.host_triangles(s), env_rgba=env, ctx=ctx)
    return s, d


def params(s, w, h, spp, depth, **kw):
    c = mcpt.Camera.from_buffer_copy(bytes(s.camera))
    c.image_width, c.image_height, c.aspect_ratio = w, h, w / float(h)
    mcpt.camera_initialize(c)
    return mcpt.render_params(c, w, h, spp, depth, seed=77, **kw)


def render(ctx, d, b, p):
    """The image, or the status of the call that was refused."""
    if p.rng == mcpt.RNG_XORWOW:
        mcpt.check(ctx.lib.mc_rng_reset(ctx.handle, p.width, p.height, 77))
    acc = torch.zeros(p.width * p.height * 3, dtype=torch.float32, device="cuda")
    try:
        mcpt.check(ctx.lib.mc_render_wavefront(ctx.handle, b.handle, C.byref(d.view), C.byref(p), acc.data_ptr(), None))
    except mcpt.McError as e:
        return e.status
    return acc.cpu().numpy()


def same(a, b):
    return np.array_equal(a, b) if isinstance(a, np.ndarray) and isinstance(b, np.ndarray) else a is b or a == b


def in_turn(ctx, d, b, s, size, options):
    """Renders the calls one after another as graphs; each must give what it gives without one."""
    w, h, spp, depth = size
    got = [render(ctx, d, b, params(s, w, h, spp, depth, use_graph=True, **o)) for o in options]
    want = [render(ctx, d, b, params(s, w, h, spp, depth, **o)) for o in options]
    for o, g, x in zip(options, got, want):
        assert same(g, x), o
    return want


@pytest.mark.parametrize("size,kw", [((64, 48, 1, 8), {}), ((64, 48, 1, 8), dict(rng=mcpt.RNG_XORWOW)),
                                     ((300, 256, 1, 6), {})])
def test_stack_and_block_size(ctx, size, kw):
    s, d = member(ctx, 3000)
    b = mcpt.Bvh(ctx, d.view, layout=mcpt.LAYOUT_WIDE4)
    want = in_turn(ctx, d, b, s, size, [dict(kw, stack_entries=1), dict(kw), dict(kw, stack_entries=2),
                                        dict(kw, stack_entries=64), dict(kw, trace_threads=128),
                                        dict(kw, trace_threads=256)])
    assert want[0] == STACK_OVERFLOW and isinstance(want[1], np.ndarray)
    b.close()
    mcpt.free_scene(s)


@pytest.mark.parametrize("rng", [mcpt.RNG_PHILOX, mcpt.RNG_XORWOW])
def test_queue_capacity(ctx, rng):
    s, d = member(ctx, 3000)
    b = mcpt.Bvh(ctx, d.view, layout=mcpt.LAYOUT_WIDE4)
    want = in_turn(ctx, d, b, s, (64, 48, 1, 8), [dict(rng=rng, queue_capacity=100), dict(rng=rng, queue_capacity=4000),
                                                  dict(rng=rng), dict(rng=rng, queue_capacity=50)])
    assert want[0] == want[3] == QUEUE_OVERFLOW and isinstance(want[1], np.ndarray)
    b.close()
    mcpt.free_scene(s)


@pytest.mark.parametrize("rng,depth", [(mcpt.RNG_XORWOW, 8), (mcpt.RNG_PHILOX, 1), (mcpt.RNG_PHILOX, 8)])
def test_environment_sampling(ctx, rng, depth):
    env = np.random.default_rng(1).uniform(0, 2, (16, 32, 4)).astype(np.float32)
    s, d = member(ctx, 3000, env=env)
    b = mcpt.Bvh(ctx, d.view, layout=mcpt.LAYOUT_WIDE4)
    cdf, alias = (dict(rng=rng, env_sampling=m) for m in (0, 1))
    want = in_turn(ctx, d, b, s, (64, 48, 1, depth), [cdf, alias, cdf])
    assert not np.array_equal(want[0], want[1])
    b.close()
    mcpt.free_scene(s)


def test_batches_of_other_trees(ctx):
    """Two batches of equal image sizes: trees of six triangles, whose rays
    need at most eight stack entries, then trees that need more."""
    sets = []
    for few in (True, False):
        scenes = [mcpt.generate_scene(mcpt.SCENE_BATCH_MEMBER, variant=v, seed=3, triangle_target=20000) for v in range(2)]
        tris = [mcpt.host_triangles(s) for s in scenes]
        if few:
            tris = [(mcpt.Triangle * 6)(*list(t)[:6]) for t in tris]
        devs = [mcpt.DeviceScene(t, ctx=ctx) for t in tris]
        batch = mcpt.BatchBvh(ctx, [d.view for d in devs])
        accs = [torch.zeros(48 * 48 * 3, dtype=torch.float32, device="cuda") for _ in devs]
        sets.append((scenes, devs, batch, accs))

    def run(k, graph, **kw):
        scenes, devs, batch, accs = sets[k]
        for a in accs:
            a.zero_()
        items = [mcpt.BatchItem(d.view, params(s, 48, 48, 2, 6, **kw), a.data_ptr())
                 for s, d, a in zip(scenes, devs, accs)]
        batch.render(items, use_graph=graph)
        return [a.cpu().numpy() for a in accs]
    run(0, False, stack_entries=8)
    with pytest.raises(mcpt.McError) as e:
        run(1, False, stack_entries=8)
    assert e.value.status == STACK_OVERFLOW
    graphs = [run(k, True) for k in (0, 1, 0)]
    plain = [run(k, False) for k in (0, 1, 0)]
    for g, x in zip(graphs, plain):
        for a, b in zip(g, x):
            assert np.array_equal(a, b)
    assert all(a.any() for a in graphs[1])
    for scenes, _, batch, _ in sets:
        batch.close()
        for s in scenes:
            mcpt.free_scene(s)


def test_grown_medium_buffers(ctx):
    """A larger render with density grids between two replays moves the buffers of the medium crossings."""
    s0, d0 = member(ctx, 300)
    b0 = mcpt.Bvh(ctx, d0.view, layout=mcpt.LAYOUT_WIDE4)
    dens, org = mcpt.fog_sphere(60.0, 6.0)
    g, hd = mcpt.volume_grid_create(ctx, dens * 0.02, tuple(np.asarray(org, np.float32) + np.float32([0, 100, -40])), 6.0)
    s = mcpt.SceneHost()
    mcpt.check(ctx.lib.mc_scene_cloud(g, C.byref(hd), 1, C.byref(s)))
    d = mcpt.DeviceScene(mcpt.host_triangles(s), spheres=mcpt.host_spheres(s), ctx=ctx)
    b = mcpt.Bvh(ctx, d.view, layout=mcpt.LAYOUT_WIDE4)
    render(ctx, d0, b0, params(s0, 200, 200, 1, 4))  # the wave's own buffers reach their size here
    small = dict(rng=mcpt.RNG_XORWOW)
    first = render(ctx, d, b, params(s, 40, 40, 1, 8, use_graph=True, **small))
    render(ctx, d, b, params(s, 160, 160, 1, 8, **small))
    again = render(ctx, d, b, params(s, 40, 40, 1, 8, use_graph=True, **small))
    assert first.any() and np.array_equal(first, again)
    assert np.array_equal(first, render(ctx, d, b, params(s, 40, 40, 1, 8, **small)))
    b.close()
    b0.close()
    mcpt.free_scene(s)
    mcpt.free_scene(s0)
    mcpt.volume_grid_destroy(g)
