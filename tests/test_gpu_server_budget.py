"""The server charges a scene for the device memory its tree holds: the leaf
records, the exported order, the 4-wide nodes and, for trees that have them,
the octant nodes."""
import pytest

import mcpt

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ctx():
    c = mcpt.Context(0)
    yield c
    c.close()


def scene(ctx, target, kind=mcpt.SCENE_BATCH_MEMBER):
    s = mcpt.generate_scene(kind, variant=4, seed=3, triangle_target=target)
    return s, mcpt.DeviceScene(mcpt.host_triangles(s), spheres=mcpt.host_spheres(s), ctx=ctx)


@pytest.mark.parametrize("kind,target", [(mcpt.SCENE_CORNELL_SPHERES, 0), (mcpt.SCENE_BATCH_MEMBER, 300),
                                         (mcpt.SCENE_BATCH_MEMBER, 30000), (mcpt.SCENE_BATCH_MEMBER, 300000),
                                         (mcpt.SCENE_BATCH_MEMBER, 2000000)])
def test_charge_is_what_the_tree_holds(ctx, kind, target):
    s, d = scene(ctx, target, kind)
    b = mcpt.Bvh(ctx, d.view, layout=mcpt.LAYOUT_WIDE4)
    i = b.info()
    n, wide = i.primitive_count, i.node_bytes
    octant = wide // 128 * 192
    b.close()
    srv = mcpt.Server(ctx)
    srv.add_scene(d)
    charged = srv.stats().scene_bytes
    srv.close()
    mcpt.free_scene(s)
    # 64-byte records; code, id and type; parents of n leaves and n - 1 nodes; each array ends on 256 bytes
    holds = n * 64 + n * 12 + (2 * n - 1) * 4 + wide + (octant if octant <= 48 << 20 else 0)
    assert holds <= charged <= holds + 6 * 256


def test_many_scenes_stay_within_their_charge(ctx):
    """120 resident scenes: the device memory they take, measured, against
    their charge. The pool maps memory 32 MiB at a time, and the last build's
    work (270 bytes a primitive) may lie beside the trees."""
    s, d = scene(ctx, 30000)
    n = s.triangle_count
    mcpt.Context(0).close()  # a context that closes gives the pool's unused memory back
    srv = mcpt.Server(ctx)
    srv.add_scene(d)
    torch.cuda.synchronize()
    free0, charge0 = torch.cuda.mem_get_info()[0], srv.stats().scene_bytes
    for _ in range(120):
        srv.add_scene(d)
    torch.cuda.synchronize()
    taken = free0 - torch.cuda.mem_get_info()[0]
    assert taken <= srv.stats().scene_bytes - charge0 + (32 << 20) + 270 * n
    srv.close()
    mcpt.free_scene(s)
