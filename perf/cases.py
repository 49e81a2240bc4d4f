"""What the framework's speed is measured on: calls a user's program makes through the public
binding (monocuda-pt_b200/mcpt.py over include/mc_abi.h), from the smallest preview to the
headline frame.

A case is a dict of plain values; "kind" selects the work:

  frame     a scene that is resident (arrays ingested, BVH built): render a frame from a zeroed
            accumulation buffer, resolve it (auto exposure, ACES, sRGB, 8 bits)
  guided    a guided frame of the aperture room with the guide training online
  rays      a set of rays against a resident scene: closest hits or occlusion
  rebuild   a moved scene: BVH from the device arrays, the sorted order, and a first set of rays
  batch     several scenes built in one pass and rendered in shared waves
  host      host triangles in, a PNG file out (upload, ingestion, build, render, read-back, encode)
  infer     the guide MLP's forward pass: vMF mixtures for a set of queries
  gradient  its forward and backward pass: loss and parameter gradients of a set of records

Everything random comes from the seed: the geometry, the renders' random numbers, rays, queries,
records and weights.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "monocuda-pt_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import mcpt  # noqa: E402

_ctx = None


def _context():
    """One context per process, as a program that renders keeps one."""
    global _ctx
    if _ctx is None:
        _ctx = mcpt.Context(0)
    return _ctx


def listed():
    return [
        # an interactive preview or a thumbnail: one sample of a few thousand pixels, all latency
        {"name": "preview_64x48", "kind": "frame", "scene": "cornell_boxes", "size": 0, "width": 64, "height": 48, "spp": 1,
         "depth": 8, "rng": "philox", "layout": "wide4"},
        # the reference's demo frame (600 x 600, depth 20, its Cornell scene with moving, metal and
        # glass spheres and fog) at a progressive renderer's few samples per update
        {"name": "spheres_600x600", "kind": "frame", "scene": "cornell_spheres", "size": 0, "width": 600, "height": 600,
         "spp": 4, "depth": 20, "rng": "philox", "layout": "wide4"},
        # the headline frame: 3.9M triangles, sky, medium box, 1080p, depth 8, 16 spp
        {"name": "icospheres_1080p", "kind": "frame", "scene": "icospheres", "size": 8, "width": 1920, "height": 1080,
         "spp": 16, "depth": 8, "rng": "philox", "layout": "wide4"},
        # the reference's cloud frame: a density grid, the camera's 333 x 180, depth 1000, one progressive sample
        {"name": "cloud_333x180", "kind": "frame", "scene": "cloud", "size": 48, "width": 333, "height": 180, "spp": 1,
         "depth": 1000, "rng": "philox", "layout": "wide4"},
        # learned guiding as the render server runs it: a resident room, training online
        {"name": "guided_512x512", "kind": "guided", "scene": "room", "size": 0, "width": 512, "height": 512, "spp": 4,
         "depth": 8},
        # baking and visibility queries: a million scattered rays against a mid-sized scene
        {"name": "rays_1m", "kind": "rays", "query": "closest", "layout": "wide4", "triangles": 500000, "rays": 1 << 20},
        # picking, collision or line-of-sight tests: an odd, small set on the default layout
        {"name": "rays_5003_any", "kind": "rays", "query": "any", "layout": "binary", "triangles": 20011, "rays": 5003},
        # dynamic geometry: rebuild a large scene, then query it
        {"name": "rebuild_1m", "kind": "rebuild", "layout": "wide4", "triangles": 1000003, "rays": 65536},
        # many small jobs at once (thumbnails, data generation)
        {"name": "batch_16", "kind": "batch", "scenes": 16, "triangles": 6000, "size": 128, "spp": 4},
        # the command-line use: host scene in, image file out
        {"name": "host_frame", "kind": "host", "triangles": 30000, "width": 640, "height": 360, "spp": 4, "depth": 8},
        # the guide's forward pass on the vertices of a 512 x 512 bounce
        {"name": "infer_262144", "kind": "infer", "n": 262144},
        # one training batch of the guide
        {"name": "gradient_65536", "kind": "gradient", "n": 65536},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "guided", "rays", "rays", "rebuild", "batch", "host", "infer", "gradient"])
    if kind == "frame":
        scene = rng.choice(["cornell_boxes", "cornell_spheres", "icospheres", "member", "cloud"])
        if scene == "cloud":
            w = _log(rng, 48, 333)
            return {"kind": kind, "scene": scene, "size": _log(rng, 16, 64), "width": w, "height": max(1, 180 * w // 333),
                    "spp": rng.choice([1, 2]), "depth": 1000, "rng": "philox", "layout": "wide4"}
        w = _log(rng, 33, 1920)
        return {"kind": kind, "scene": scene,
                "size": rng.choice([4, 5, 6, 7]) if scene == "icospheres" else _log(rng, 1000, 200000) if scene == "member" else 0,
                "width": w, "height": max(1, int(w * rng.uniform(0.5, 1.0))), "spp": _log(rng, 1, 16),
                "depth": rng.choice([1, 4, 8, 8, 20]), "rng": rng.choice(["philox"] * 5 + ["xorwow"]),
                "layout": rng.choice(["wide4"] * 4 + ["binary", "wide4q"])}
    if kind == "guided":
        w = _log(rng, 65, 700)
        return {"kind": kind, "scene": "room", "size": 0, "width": w, "height": max(1, int(w * rng.uniform(0.5, 1.0))),
                "spp": _log(rng, 1, 8), "depth": rng.choice([4, 8])}
    if kind == "rays":
        return {"kind": kind, "query": rng.choice(["closest", "any"]), "layout": rng.choice(["wide4", "wide4", "binary", "wide4q"]),
                "triangles": _log(rng, 100, 1000000), "rays": _log(rng, 1, 4 << 20)}
    if kind == "rebuild":
        return {"kind": kind, "layout": rng.choice(["wide4", "wide4", "binary", "wide4q"]),
                "triangles": _log(rng, 36, 2000000), "rays": _log(rng, 1000, 100000)}
    if kind == "batch":
        return {"kind": kind, "scenes": _log(rng, 2, 48), "triangles": _log(rng, 1000, 30000), "size": _log(rng, 32, 256),
                "spp": _log(rng, 1, 8)}
    if kind == "host":
        w = _log(rng, 64, 1280)
        return {"kind": kind, "triangles": _log(rng, 1000, 200000), "width": w, "height": max(1, int(w * rng.uniform(0.5, 1.0))),
                "spp": _log(rng, 1, 8), "depth": rng.choice([4, 8])}
    if kind == "infer":
        return {"kind": kind, "n": _log(rng, 1, 1 << 20)}
    return {"kind": kind, "n": _log(rng, 100, 1 << 18)}


# ---------------------------------------------------------------------------
# Scenes
# ---------------------------------------------------------------------------
_LAYOUTS = {"binary": mcpt.LAYOUT_BINARY, "wide4": mcpt.LAYOUT_WIDE4, "wide4q": mcpt.LAYOUT_WIDE4Q}


class _Resident:
    """A scene on the device with its tree, released when the program drops it."""

    def __init__(self, ctx, host, layout="wide4", grid=None):
        self.ctx, self.grid = ctx, grid
        self.camera = mcpt.Camera.from_buffer_copy(bytes(host.camera))
        self.scene = mcpt.DeviceScene(mcpt.host_triangles(host), spheres=mcpt.host_spheres(host), env_rgba=mcpt.host_env(host),
                                      env_intensity=host.env_intensity, ctx=ctx)
        self.bvh = mcpt.Bvh(ctx, self.scene.view, layout=_LAYOUTS[layout])
        mcpt.free_scene(host)

    def __del__(self):
        self.bvh.close()
        self.scene.close()
        if self.grid:
            mcpt.volume_grid_destroy(self.grid)


def _camera(cam, width, height, depth, spp):
    cam = mcpt.Camera.from_buffer_copy(bytes(cam))
    cam.image_width = width
    cam.image_height = height
    cam.aspect_ratio = width / float(height)
    cam.max_depth = depth
    cam.samples_per_pixel = spp
    return mcpt.camera_initialize(cam)


def _cloud(ctx, size, seed):
    """The cloud scene around a lumpy density grid of size^3 voxels."""
    g = np.random.default_rng(seed)
    x = np.linspace(-1.0, 1.0, size, dtype=np.float32)
    z, y, x = np.meshgrid(x, x, x, indexing="ij")
    lumps = np.zeros_like(x)
    for _ in range(6):
        c, s = g.uniform(-0.5, 0.5, 3), g.uniform(0.25, 0.45)
        lumps = np.maximum(lumps, 1.0 - np.sqrt((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2) / s)
    density = np.clip(lumps * 2.0, 0.0, 1.0) * g.uniform(0.6, 1.0, lumps.shape).astype(np.float32)
    voxel = 160.0 / size
    origin = (-80.0, 20.0, -120.0)
    grid, header = mcpt.volume_grid_create(ctx, density.astype(np.float32), origin, voxel)
    host = mcpt.SceneHost()
    mcpt.check(ctx.lib.mc_scene_cloud(grid, C.byref(header), 1, C.byref(host)))
    return host, grid


def _host_scene(ctx, case, seed):
    """(host scene, density grid or None)"""
    scene, seed = case["scene"], seed % (1 << 20) + 2
    if scene == "cloud":
        return _cloud(ctx, case["size"], seed)
    if scene == "cornell_boxes":
        return mcpt.generate_scene(mcpt.SCENE_CORNELL_BOXES), None
    if scene == "cornell_spheres":
        return mcpt.generate_scene(mcpt.SCENE_CORNELL_SPHERES, seed=seed), None
    if scene == "icospheres":
        return mcpt.generate_scene(mcpt.SCENE_DISPLACED_ICOSPHERES, variant=case["size"], seed=seed), None
    if scene == "room":
        return mcpt.generate_scene(mcpt.SCENE_GUIDING_ROOM, seed=seed), None
    return mcpt.generate_scene(mcpt.SCENE_BATCH_MEMBER, variant=seed & 1, seed=seed, triangle_target=case["size"]), None


def _terrain(n, seed):
    """n triangles [n, 9], float32: a bumpy height field over [-1, 1]^2, loose triangles above it and
    a quad below it, which every downward ray inside the square hits at the latest."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    side = max(1, int(math.sqrt(0.8 * n / 2)))
    i = torch.arange(side + 1, device="cuda", dtype=torch.float32) * (2.0 / side) - 1.0
    z, x = torch.meshgrid(i, i, indexing="ij")
    ph = torch.rand(8, 3, device="cuda", generator=g)
    y = torch.zeros_like(x)
    for k in range(8):
        f = 2.0 ** (1 + k * 0.75)
        a = 6.2831853 * ph[k, 0]
        y = y + (0.25 / f) * torch.sin(f * (x * torch.cos(a) + z * torch.sin(a)) * 3.0 + 6.2831853 * ph[k, 1])
    p = torch.stack([x, y, z], -1)
    a, b, c, d = p[:-1, :-1], p[:-1, 1:], p[1:, :-1], p[1:, 1:]
    ground = torch.cat([torch.cat([a, c, b], -1).reshape(-1, 9), torch.cat([b, c, d], -1).reshape(-1, 9)])
    rest = n - ground.shape[0]
    ctr = torch.rand(max(rest, 0), 1, 3, device="cuda", generator=g) * torch.tensor([1.96, 0.6, 1.96], device="cuda") + \
        torch.tensor([-0.98, 0.1, -0.98], device="cuda")
    off = (torch.rand(max(rest, 0), 3, 3, device="cuda", generator=g) - 0.5) * (2.0 / side)
    floor = torch.tensor([[-3, -0.95, -3, -3, -0.95, 3, 3, -0.95, -3], [3, -0.95, -3, -3, -0.95, 3, 3, -0.95, 3]],
                         device="cuda", dtype=torch.float32)
    tris = torch.cat([floor, ground, (ctr + off).reshape(-1, 9)])[:n]
    return tris[torch.randperm(tris.shape[0], device="cuda", generator=g)].contiguous()


class _Triangles:
    """Device triangles handed to the library as full records (mc_scene_ingest)."""

    def __init__(self, ctx, verts):
        n = verts.shape[0]
        full = torch.zeros(n, 56, dtype=torch.float32, device="cuda")  # 224-byte records, lambertian
        full[:, :9] = verts
        self.hot = torch.empty(n * 36, dtype=torch.uint8, device="cuda")
        self.cold = torch.empty(n * 192, dtype=torch.uint8, device="cuda")
        self.lights = torch.empty(64, dtype=torch.uint8, device="cuda")
        mcpt.check(ctx.lib.mc_scene_ingest(ctx.handle, full.data_ptr(), n, None, 0, self.hot.data_ptr(), self.cold.data_ptr(),
                                           None, None, None))
        v = mcpt.SceneView()
        v.tri_hot, v.tri_cold, v.triangle_count = self.hot.data_ptr(), self.cold.data_ptr(), n
        v.lights = self.lights.data_ptr()
        self.view, self.n = v, n


def _rays(n, seed):
    """Rays [7, n] from above the terrain toward points scattered below it, in no order."""
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    o = torch.rand(3, n, device="cuda", generator=g) * 1.8 - 0.9
    o[1] = 0.5 + 0.7 * torch.rand(n, device="cuda", generator=g)
    t = torch.rand(3, n, device="cuda", generator=g) * 1.8 - 0.9
    t[1] = -1.0
    d = t - o
    d = d / d.square().sum(0, keepdim=True).sqrt()
    return torch.cat([o, d, torch.full((1, n), 0.5, device="cuda")]).contiguous()


# ---------------------------------------------------------------------------
# The guide MLP's inputs
# ---------------------------------------------------------------------------
def _unit(v):
    return v / v.square().sum(-1, keepdim=True).sqrt()


def _weights(seed):
    """Flat parameters of a guide, spread as an initialised and somewhat trained one's."""
    g = torch.Generator().manual_seed(seed + 3)
    parts = []
    for fan_out, fan_in, gain in ((64, 144, 1.0), (64, 64, 1.0), (64, 64, 1.0), (40, 64, 0.3)):
        parts.append((torch.rand(fan_out * fan_in, generator=g) * 2 - 1) * math.sqrt(6.0 / fan_in) * gain)
        parts.append((torch.rand(fan_out, generator=g) * 2 - 1) * 0.1)
    parts[-1][32:] += 1.0
    return torch.cat(parts).to(torch.float32)


def _guide(ctx, seed):
    guide = mcpt.Guide(ctx, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0), seed=seed % 1000 + 1)
    guide.set_params(_weights(seed).numpy())
    return guide


def _queries(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed + 5)
    pos = torch.rand(n, 3, device="cuda", generator=g)
    return torch.cat([pos, _unit(torch.randn(n, 3, device="cuda", generator=g))], -1).contiguous()


def _records(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed + 7)
    pos = torch.rand(n, 3, device="cuda", generator=g)
    nrm = _unit(torch.randn(n, 3, device="cuda", generator=g))
    nxt = _unit(nrm + _unit(torch.randn(n, 3, device="cuda", generator=g)) * 0.98)
    w = torch.exp(torch.randn(n, 1, device="cuda", generator=g)) / n
    return torch.cat([pos, nrm, nxt, w], -1).contiguous()


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    ctx = _context()
    s = {"case": case, "ctx": ctx}
    kind = case["kind"]
    if kind in ("frame", "guided"):
        W, H = case["width"], case["height"]
        host, grid = _host_scene(ctx, case, seed)
        bounds = None
        if kind == "guided":
            raw = np.frombuffer(mcpt.host_triangles(host), dtype=np.uint8).reshape(host.triangle_count, 224)
            v = raw[:, :36].copy().view(np.float32).reshape(-1, 3)
            bounds = [tuple(float(x) for x in v.min(0)), tuple(float(x) for x in v.max(0))]
        s["resident"] = _Resident(ctx, host, case.get("layout", "wide4"), grid)
        s["params"] = mcpt.render_params(_camera(s["resident"].camera, W, H, case["depth"], case["spp"]), W, H, case["spp"],
                                         case["depth"], seed=seed + 17,
                                         rng=mcpt.RNG_XORWOW if case.get("rng") == "xorwow" else mcpt.RNG_PHILOX)
        s["accum"] = torch.zeros(H * W * 3, dtype=torch.float32, device="cuda")
        s["rgb"] = torch.empty(H * W * 3, dtype=torch.uint8, device="cuda")
        if kind == "guided":
            s["guide"] = mcpt.Guide(ctx, bounds[0], bounds[1], seed=seed % 1000 + 1)
    elif kind == "rays":
        s["scene"] = _Triangles(ctx, _terrain(case["triangles"], seed))
        s["bvh"] = mcpt.Bvh(ctx, s["scene"].view, layout=_LAYOUTS[case["layout"]])
        s["rays"] = _rays(case["rays"], seed)
        s["tmax"] = torch.full((case["rays"],), 0.8, device="cuda")
        s["hits"] = torch.empty(case["rays"], 4, dtype=torch.int32, device="cuda")
        s["occluded"] = torch.empty(case["rays"], dtype=torch.int32, device="cuda")
    elif kind == "rebuild":
        s["scene"] = _Triangles(ctx, _terrain(case["triangles"], seed))
        s["rays"] = _rays(case["rays"], seed)
        s["hits"] = torch.empty(case["rays"], 4, dtype=torch.int32, device="cuda")
        s["codes"] = torch.empty(case["triangles"], dtype=torch.int32, device="cuda")
        s["ids"] = torch.empty(case["triangles"], dtype=torch.int32, device="cuda")
    elif kind == "batch":
        s["scenes"], s["items"], s["accums"], views = [], [], [], []
        for i in range(case["scenes"]):
            host = mcpt.generate_scene(mcpt.SCENE_BATCH_MEMBER, variant=i, seed=seed % (1 << 20) + 3,
                                       triangle_target=max(1000, case["triangles"] * (i % 4 + 1) // 2))
            d = mcpt.DeviceScene(mcpt.host_triangles(host), ctx=ctx)
            W = max(16, case["size"] * (3 - i % 3) // 3)
            acc = torch.zeros(W * W * 3, dtype=torch.float32, device="cuda")
            p = mcpt.render_params(_camera(host.camera, W, W, 8, case["spp"]), W, W, case["spp"], 8, seed=seed + i)
            mcpt.free_scene(host)
            s["scenes"].append(d)
            s["accums"].append(acc)
            s["items"].append(mcpt.BatchItem(d.view, p, acc.data_ptr()))
            views.append(d.view)
        s["views"] = views
    elif kind == "host":
        W, H = case["width"], case["height"]
        s["host"] = _HostScene(case["triangles"], seed)
        s["params"] = mcpt.render_params(_camera(s["host"].scene.camera, W, H, case["depth"], case["spp"]), W, H, case["spp"],
                                         case["depth"], seed=seed + 17)
    elif kind == "infer":
        s["guide"] = _guide(ctx, seed)
        s["queries"] = _queries(case["n"], seed)
        s["mixtures"] = torch.empty(case["n"], mcpt.GUIDE_OUTPUTS, dtype=torch.float32, device="cuda")
    else:
        s["guide"] = _guide(ctx, seed)
        s["records"] = _records(case["n"], seed)
        s["grad"] = torch.empty(mcpt.GUIDE_PARAM_COUNT, dtype=torch.float32, device="cuda")
    return s


class _HostScene:
    """A generated scene in host memory, freed when the program drops it."""

    def __init__(self, triangles, seed):
        self.scene = mcpt.generate_scene(mcpt.SCENE_BATCH_MEMBER, variant=seed & 1, seed=seed % (1 << 20) + 3,
                                         triangle_target=triangles)

    def __del__(self):
        mcpt.free_scene(self.scene)


def run(state):
    return _RUN[state["case"]["kind"]](state, state["case"], state["ctx"])


def _run_frame(s, case, ctx):
    p, r = s["params"], s["resident"]
    st = mcpt.RenderStats()
    s["accum"].zero_()
    if case["rng"] == "xorwow":
        mcpt.check(ctx.lib.mc_rng_reset(ctx.handle, p.width, p.height, p.seed))
    mcpt.check(ctx.lib.mc_render_wavefront(ctx.handle, r.bvh.handle, C.byref(r.scene.view), C.byref(p), s["accum"].data_ptr(),
                                           C.byref(st)))
    mcpt.image_encode(ctx, s["accum"].data_ptr(), p.width, p.height, p.spp, tonemap=mcpt.TONEMAP_ACES, exposure=0.0,
                      device_out=s["rgb"].data_ptr())
    return {"accum": s["accum"], "rgb": s["rgb"], "extend_rays": st.extend_rays, "shadow_rays": st.shadow_rays}


def _run_guided(s, case, ctx):
    p, r = s["params"], s["resident"]
    st = mcpt.RenderStats()
    s["accum"].zero_()
    mcpt.check(ctx.lib.mc_render_guided(ctx.handle, r.bvh.handle, C.byref(r.scene.view), C.byref(p), s["guide"].handle, 1,
                                        s["accum"].data_ptr(), C.byref(st)))
    return {"accum": s["accum"], "params": s["guide"].get_params(), "extend_rays": st.extend_rays, "shadow_rays": st.shadow_rays}


def _closest(s, ctx, bvh, n):
    mcpt.check(ctx.lib.mc_trace_closest(ctx.handle, bvh.handle, C.byref(s["scene"].view), s["rays"].data_ptr(), n,
                                        mcpt.ISECT_REFERENCE, s["hits"].data_ptr()))
    return {"t": s["hits"][:, 0].view(torch.float32), "hit": s["hits"][:, 1:]}


def _run_rays(s, case, ctx):
    if case["query"] == "closest":
        return _closest(s, ctx, s["bvh"], case["rays"])
    mcpt.check(ctx.lib.mc_trace_any(ctx.handle, s["bvh"].handle, C.byref(s["scene"].view), s["rays"].data_ptr(),
                                    s["tmax"].data_ptr(), case["rays"], mcpt.ISECT_REFERENCE, s["occluded"].data_ptr()))
    return {"occluded": s["occluded"]}


def _run_rebuild(s, case, ctx):
    bvh = mcpt.Bvh(ctx, s["scene"].view, layout=_LAYOUTS[case["layout"]])
    bvh.export(codes=s["codes"], ids=s["ids"])
    out = _closest(s, ctx, bvh, case["rays"])
    bvh.close()
    return dict(out, codes=s["codes"], ids=s["ids"])


def _run_batch(s, case, ctx):
    for a in s["accums"]:
        a.zero_()
    batch = mcpt.BatchBvh(ctx, s["views"])
    st = batch.render(s["items"])
    batch.close()
    return {"accums": s["accums"], "extend_rays": st.extend_rays, "shadow_rays": st.shadow_rays}


def _run_host(s, case, ctx):
    p, scene, lib = s["params"], s["host"].scene, ctx.lib
    accum = np.zeros(p.width * p.height * 3, np.float32)
    st = mcpt.RenderStats()
    mcpt.check(lib.mc_render_host(ctx.handle, C.addressof(scene.triangles.contents), scene.triangle_count, None, 0, None,
                                  C.byref(p), accum.ctypes.data, C.byref(st)))
    opts = mcpt.ImageOptions(mcpt.IMAGE_PNG, mcpt.TONEMAP_REINHARD, 1.0, 0)
    size = C.c_int64()
    mcpt.check(lib.mc_image_encode_host(ctx.handle, accum.ctypes.data, p.width, p.height, p.spp, C.byref(opts), None, C.byref(size), None))
    png = np.empty(size.value, np.uint8)
    mcpt.check(lib.mc_image_encode_host(ctx.handle, accum.ctypes.data, p.width, p.height, p.spp, C.byref(opts), png.ctypes.data,
                                        C.byref(size), None))
    return {"accum": accum, "png": png, "extend_rays": st.extend_rays, "shadow_rays": st.shadow_rays}


def _run_infer(s, case, ctx):
    mcpt.check(ctx.lib.mc_guide_infer(s["guide"].handle, s["queries"].data_ptr(), case["n"], s["mixtures"].data_ptr()))
    return {"mixtures": s["mixtures"]}


def _run_gradient(s, case, ctx):
    loss = C.c_double()
    mcpt.check(ctx.lib.mc_guide_gradient(s["guide"].handle, s["records"].data_ptr(), case["n"], s["grad"].data_ptr(),
                                         C.byref(loss)))
    return {"grad": s["grad"], "loss": loss.value}


_RUN = {"frame": _run_frame, "guided": _run_guided, "rays": _run_rays, "rebuild": _run_rebuild, "batch": _run_batch,
        "host": _run_host, "infer": _run_infer, "gradient": _run_gradient}


# ---------------------------------------------------------------------------
# work / exact
# ---------------------------------------------------------------------------
def _scene_triangles(case):
    return {"cornell_boxes": 36, "cornell_spheres": 156, "icospheres": 60 * 4 ** case["size"], "cloud": 5, "room": 205300,
            "member": case["size"]}[case["scene"]]


def _trace_flops(rays, triangles):
    """Slab tests on a path from the root to one leaf of a 4-wide tree and one triangle test."""
    return rays * (math.log(max(triangles, 4), 4) * 4 * 12 + 60)


def work(case):
    kind = case["kind"]
    if kind in ("frame", "guided"):
        paths = case["width"] * case["height"] * case["spp"]
        tris = _scene_triangles(case)
        # a path casts about two extend and one shadow ray; the scene's vertices are read, the image written
        pixels = case["width"] * case["height"]
        flops = _trace_flops(3 * paths, tris)
        return {"bytes": min(tris, 3 * paths) * 36 + pixels * 15, "flops": flops + (paths * 39936 if kind == "guided" else 0)}
    if kind == "rays":
        out = 16 if case["query"] == "closest" else 4
        return {"bytes": case["rays"] * (28 + out) + min(case["triangles"], case["rays"]) * 36,
                "flops": _trace_flops(case["rays"], case["triangles"])}
    if kind == "rebuild":
        # vertices in; sorted order, primitive records and a 4-wide node per two primitives out
        return {"bytes": case["triangles"] * (36 + 8 + 48 + 64) + case["rays"] * 44,
                "flops": _trace_flops(case["rays"], case["triangles"])}
    if kind == "batch":
        paths = sum(max(16, case["size"] * (3 - i % 3) // 3) ** 2 * case["spp"] for i in range(case["scenes"]))
        tris = sum(max(1000, case["triangles"] * (i % 4 + 1) // 2) for i in range(case["scenes"]))
        return {"bytes": tris * 148 + paths // case["spp"] * 12, "flops": _trace_flops(3 * paths, case["triangles"])}
    if kind == "host":
        paths = case["width"] * case["height"] * case["spp"]
        return {"bytes": case["triangles"] * 224 + case["width"] * case["height"] * 15,
                "flops": _trace_flops(3 * paths, case["triangles"])}
    if kind == "infer":
        return {"bytes": case["n"] * (24 + 160) + 20200 * 4, "flops": case["n"] * 39936}
    return {"bytes": case["n"] * 40 + 2 * 20200 * 4, "flops": case["n"] * 101376}


def _net64(flat, x):
    """The guide MLP in 64 bits: raw outputs for coordinates x [n, 6] in the unit box."""
    f = 2.0 ** torch.arange(12, dtype=torch.float64, device=x.device)
    a = math.pi * x[:, :, None] * f
    h = torch.stack([torch.sin(a), torch.cos(a)], -1).reshape(x.shape[0], 144)
    at = 0
    for fan_out, fan_in in ((64, 144), (64, 64), (64, 64), (40, 64)):
        w = flat[at:at + fan_out * fan_in].reshape(fan_out, fan_in)
        b = flat[at + fan_out * fan_in:at + fan_out * fan_in + fan_out]
        at += fan_out * fan_in + fan_out
        h = h @ w.T + b
        if fan_out == 64:
            h = torch.relu(h)
    return h


def _mixture64(y, direction):
    """Weights, unit means (anchored to the direction input) and concentrations."""
    mean = y[:, 8:32].reshape(-1, 8, 3) + 1.5 * direction[:, None, :]
    return torch.softmax(y[:, :8], -1), _unit(mean), torch.exp(y[:, 32:].clamp(math.log(0.01), math.log(1000.0)))


def exact(case, seed):
    if case["kind"] == "infer":
        flat, q = _weights(seed).cuda().double(), _queries(case["n"], seed).double()
        out = []
        for part in q.split(1 << 17):
            w, mu, kappa = _mixture64(_net64(flat, part), part[:, 3:])
            out.append(torch.cat([w, mu.reshape(-1, 24), kappa], -1))
        return {"mixtures": torch.cat(out)}
    if case["kind"] == "gradient":
        flat = _weights(seed).cuda().double().requires_grad_(True)
        total = 0.0
        for r in _records(case["n"], seed).double().split(1 << 15):
            w, mu, kappa = _mixture64(_net64(flat, r[:, :6]), r[:, 3:6])
            c = (mu * r[:, None, 6:9]).sum(-1)
            q = (w * kappa / (2 * math.pi * -torch.expm1(-2 * kappa)) * torch.exp(kappa * (c - 1))).sum(-1)
            loss = -(r[:, 9] * torch.log(q)).sum()
            loss.backward()
            total += float(loss.detach())
        return {"grad": flat.grad, "loss": total}
    if (case["kind"] == "rebuild" or case.get("query") == "closest") and case["rays"] * case["triangles"] <= 1e11:
        # closest t over all triangles
        tri, rays = _terrain(case["triangles"], seed).double(), _rays(case["rays"], seed).double()
        v0, e1, e2 = tri[:, 0:3], tri[:, 3:6] - tri[:, 0:3], tri[:, 6:9] - tri[:, 0:3]
        n = torch.linalg.cross(e1, e2)
        out = []
        step = max(1, int(4e7) // tri.shape[0])
        for k in range(0, case["rays"], step):
            o, d = rays[0:3, k:k + step].T, rays[3:6, k:k + step].T
            # Cramer's rule on o + t d = v0 + u e1 + v e2, all pairs as matrix products
            det = -(d @ n.T)
            on = o @ n.T - (v0 * n).sum(-1)
            m = torch.linalg.cross(o, d)
            u = (m @ e2.T - d @ torch.linalg.cross(e2, v0).T) / det
            v = (d @ torch.linalg.cross(e1, v0).T - m @ e1.T) / det
            t = on / det
            ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 1e-4)
            out.append(torch.where(ok, t, 1e30).min(-1).values)
        out = {"t": torch.cat(out), "hit": None}
        return dict(out, codes=None, ids=None) if case["kind"] == "rebuild" else out
    return None
