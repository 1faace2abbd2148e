"""What a user of this package has it do, as cases that can be timed.

Each case is one pass through the public entry points on inputs made from a
seed: single views through the plugin classes (pipelines.py) and the stateless
C entry points, batches of uneven views, the animated many-view workload, and
the consumers of the culled lists (cluster lookup, shading, frustum culling).
Sizes, scenes and value ranges are those of scenes.py, of the tests and of the
benchmark.  The inputs are generated on the GPU, with the distributions that
scenes.py describes.  A served request runs the batch kernels on the light
sets the server keeps resident; the batch cases cover that size range.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

from hellovulkan_gb300 import camera
from hellovulkan_gb300._lib import CfBatchView, CfPBRPushConstant, check, lib, stream_handle
from hellovulkan_gb300.batch import Batch
from hellovulkan_gb300.consumer import frustum_cull, lookup_clusters, shade_clusters
from hellovulkan_gb300.pipelines import (Context, PipelineAABBGenerator, PipelineLightCulling, ResourcesClusterForward,
                                         ResourcesLight, device_view)

FOVY = math.radians(45.0)
# the grids of the batch mix, with the pixel size of a tile that gives each a matching resolution
MIX = ((8, 8, 16, 128), (16, 9, 24, 120), (24, 14, 32, 120), (32, 18, 48, 80))
PC = (1.75, 0.01, 0.0, 0.1, 0.1)  # the reference UI's push constants


def _frame(name, w, h, grid, lights, scene, near=0.1, far=2000.0, cap=150, host=False):
    return {"kind": "frame", "name": name, "w": w, "h": h, "x": grid[0], "y": grid[1], "z": grid[2], "lights": lights,
            "scene": scene, "near": near, "far": far, "cap": cap, "host": host}


def _consumer(kind, name, w, h, grid, lights, scene, depth, far, **more):
    return {"kind": kind, "name": name, "w": w, "h": h, "x": grid[0], "y": grid[1], "z": grid[2], "lights": lights,
            "scene": scene, "near": 0.1, "far": far, "cap": 150, "depth": depth, **more}


def listed():
    return [
        # the smallest view of the batch mix, its projection changing every frame (zoom): AABBs and lists, stateless
        {"kind": "zoom", "name": "zoom_tiny", "w": 1024, "h": 1024, "x": 8, "y": 8, "z": 16, "lights": 256,
         "scene": "blobs", "near": 0.1, "far": 2000.0, "cap": 150},
        # an ordinary frame of the reference app: 1920x1080, its default grid, about a thousand lights
        _frame("frame_1080p", 1920, 1080, (16, 9, 24), 1024, "box", far=1000.0),
        # a host-driven frame with nothing round about it: lights uploaded from, and lists read back to, pinned memory
        _frame("frame_host_odd", 1917, 1079, (15, 9, 23), 3001, "blobs", host=True),
        # the benchmark's headline view
        _frame("frame_1600p", 2560, 1600, (32, 18, 48), 16384, "blobs"),
        # the most lights the batch mix has, in one view: dense slices, many capped clusters
        _frame("frame_1600p_65k", 2560, 1600, (32, 18, 48), 65536, "blobs"),
        # a server's full batch (64 views) of the benchmark's uneven mix
        {"kind": "batch", "name": "batch_mix_64", "views": 64, "lights_lo": 256, "lights_hi": 65536, "mix": 3},
        # the animated workload: every light of every view moved on the device, then all views culled
        {"kind": "animate", "name": "animate_256", "views": 256, "lights": 4096, "epoch": 0},
        # Scene.frag's cluster lookup, the benchmark's depth buffer (log-uniform per pixel)
        _consumer("lookup", "lookup_1080p", 1920, 1080, (16, 9, 24), 1024, "box", "scatter", 1000.0, check=False),
        # the same with the all-lights check (the wrapper's default), at a test's size
        _consumer("lookup", "lookup_check", 480, 270, (16, 9, 24), 3000, "blobs", "scatter", 1000.0, check=True),
        # direct lighting of a G-buffer of surfaces, as a renderer has it
        _consumer("shade", "shade_surfaces", 1920, 1080, (16, 9, 24), 1024, "box", "surfaces", 1000.0),
        # the benchmark's G-buffer: every texel at its own depth
        _consumer("shade", "shade_scatter", 1920, 1080, (16, 9, 24), 1024, "box", "scatter", 1000.0),
        # frustum culling of a large scene's draw commands
        {"kind": "frustum", "name": "frustum_1m", "boxes": 1000003},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_grid(rng):
    return rng.randint(5, 40), rng.randint(4, 24), rng.randint(8, 56)


def draw(rng):
    kind = rng.choice(["zoom", "frame", "frame", "host", "batch", "animate", "lookup", "shade", "frustum"])
    grid = _draw_grid(rng)
    if kind == "batch":
        return {"kind": "batch", "views": rng.randint(3, 64), "lights_lo": 256, "lights_hi": _log_int(rng, 4096, 65536),
                "mix": rng.randint(0, 999)}
    if kind == "animate":
        return {"kind": "animate", "views": 2 * rng.randint(4, 128), "lights": _log_int(rng, 300, 4096),
                "epoch": rng.randint(0, 3)}
    if kind == "frustum":
        return {"kind": "frustum", "boxes": _log_int(rng, 10000, 4000000)}
    scene = rng.choice(["box", "blobs"])
    far = rng.choice([100.0, 1000.0, 2000.0])
    if kind in ("lookup", "shade"):
        w, h = rng.randint(320, 1920), rng.randint(200, 1080)
        depth = rng.choice(["surfaces", "scatter"])
        c = _consumer(kind, "", w, h, grid, _log_int(rng, 100, 4000), scene, depth, far)
        if kind == "lookup":
            c["check"] = w * h * c["lights"] < 4e8
    else:
        c = _frame("", rng.randint(640, 2560), rng.randint(480, 1600), grid, _log_int(rng, 16, 40000), scene, far=far,
                   cap=rng.choice([64, 150, 150, 255]), host=kind == "host")
        if kind == "zoom":
            c["kind"] = "zoom"
            del c["host"]
    del c["name"]
    return c


# ---- inputs -------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _u(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float32)


def _records(pos, radius, color):
    out = torch.zeros(pos.shape[0], 12, device="cuda")
    out[:, 0:3], out[:, 3], out[:, 4:7], out[:, 7], out[:, 8] = pos, 1.0, color, 1.0, radius
    return out


def _blob_positions(g, n, sets=1):
    """n positions for each of `sets` views, around 32 Gaussian blobs of its own."""
    lo = torch.tensor([-100.0, 0.0, -100.0], device="cuda")
    span = torch.tensor([200.0, 30.0, 200.0], device="cuda")
    centres = _u(g, sets, 32, 3) * span + lo
    which = torch.randint(0, 32, (sets, n), generator=g, device="cuda")
    pos = torch.gather(centres, 1, which[..., None].expand(sets, n, 3))
    return (pos + 8.0 * torch.randn(sets, n, 3, generator=g, device="cuda")).reshape(sets * n, 3)


def _blob_radii(g, n):
    return torch.exp(math.log(3.0) + 0.5 * torch.randn(n, generator=g, device="cuda")).clamp(0.5, 20.0)


def _lights(g, n, scene):
    if scene == "blobs":
        return _records(_blob_positions(g, n), _blob_radii(g, n), _u(g, n, 3))
    lo = torch.tensor([-20.0, 0.0, -40.0], device="cuda")
    span = torch.tensor([40.0, 15.0, 50.0], device="cuda")
    return _records(_u(g, n, 3) * span + lo, 1.0 + 4.0 * _u(g, n), _u(g, n, 3))


def _random_camera(r):
    eye = (r.uniform(-80, 80), r.uniform(2, 40), r.uniform(-80, 80))
    return camera.look_at_rh(eye, [r.uniform(-20, 20) for _ in range(3)])


def _ubo(case, view):
    return camera.cluster_forward_ubo(FOVY, case["w"], case["h"], case["near"], case["far"], view,
                                      (case["x"], case["y"], case["z"]))


def _view_matrix(case, seed):
    if case["scene"] == "box":
        return np.eye(4, dtype=np.float32)
    r = random.Random(seed)
    # the headline view's camera, moved a little from seed to seed
    return camera.look_at_rh((r.uniform(-4, 4), 10.0 + r.uniform(-2, 2), 60.0), (0.0, 0.0, 0.0))


class _State:
    """What a user's program keeps between calls."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


class _Owner:
    """The handles of one view, closed together.  The state and every tensor over the library's buffers hold it, so
    the buffers live as long as anything can read them."""

    def __init__(self, *handles):
        self.handles = handles

    def __del__(self):
        for h in self.handles:
            h.close()


def _prepare_frame(case, seed):
    g = _gen(seed)
    n, cap = case["lights"], case["cap"]
    lights = _lights(g, n, case["scene"])
    ctx = Context(0)
    rl, rc = ResourcesLight(ctx), ResourcesClusterForward(ctx)
    host = torch.empty(n, 12, dtype=torch.float32, pin_memory=True)
    host.copy_(lights)
    torch.cuda.synchronize()
    rl.add_lights(host.numpy())
    rc.create_buffers(case["x"], case["y"], case["z"], cap)
    gen, cull = PipelineAABBGenerator(ctx, rc), PipelineLightCulling(ctx, rl, rc)
    b = rc.buffers()
    cells = device_view(b.light_cells, (b.cluster_count, 2), "<i4")
    indices = device_view(b.light_indices, (b.index_capacity,), "<i4")
    indices.zero_()  # entries past the total are never written
    owner = cells.owner = indices.owner = _Owner(cull, gen, rc, rl)
    s = _State(kind="frame", ctx=ctx, rl=rl, rc=rc, gen=gen, cull=cull, ubo=_ubo(case, _view_matrix(case, seed)), n=n,
               cells=cells, indices=indices, host=host if case["host"] else None, owner=owner)
    if case["host"]:
        s.h_cells = torch.zeros(b.cluster_count, 2, dtype=torch.int32, pin_memory=True).numpy()
        s.h_indices = torch.zeros(b.index_capacity, dtype=torch.int32, pin_memory=True).numpy()
    return s


def _run_frame(s):
    if s.host is not None:
        s.rl.upload_async(s.host, s.n)
    s.gen.set_cluster_forward_ubo(s.ubo)
    s.gen.fill_command_buffer()
    s.cull.reset_global_index()
    s.cull.set_cluster_forward_ubo(s.ubo)
    s.cull.fill_command_buffer()
    if s.host is not None:
        s.rc.read_outputs(None, s.h_cells, s.h_indices)
        return s.h_cells, s.h_indices
    return s.cells, s.indices


class _Buffers:
    """Caller-owned device memory of one stateless view."""

    def __init__(self, ubo, lights, cap):
        self.ubo, self.lights, self.cap, self.n = ubo, lights, cap, lights.shape[0]
        self.clusters = ubo.sliceCountX * ubo.sliceCountY * ubo.sliceCountZ
        self.aabbs = torch.zeros(self.clusters, 8, device="cuda")
        self.cells = torch.zeros(self.clusters, 2, dtype=torch.int32, device="cuda")
        self.indices = torch.zeros(self.clusters * cap, dtype=torch.int32, device="cuda")
        self.total = torch.zeros(1, dtype=torch.int32, device="cuda")
        n = C.c_uint64()
        check(lib().cf_cull_workspace_size(C.byref(ubo), self.n, cap, C.byref(n)))
        self.ws = torch.zeros(n.value, dtype=torch.uint8, device="cuda")

    def cull(self):
        L, st = lib(), stream_handle(torch.cuda.current_stream())
        check(L.cf_generate_aabbs(C.byref(self.ubo), self.aabbs.data_ptr(), st))
        check(L.cf_cull_lights(C.byref(self.ubo), self.aabbs.data_ptr(), self.lights.data_ptr(), self.n, self.cap,
                               self.cells.data_ptr(), self.indices.data_ptr(), self.indices.numel(),
                               self.total.data_ptr(), self.ws.data_ptr(), self.ws.numel(), st))


def _prepare_zoom(case, seed):
    return _State(kind="zoom", b=_Buffers(_ubo(case, _view_matrix(case, seed)), _lights(_gen(seed), case["lights"],
                                                                                       case["scene"]), case["cap"]))


def _run_zoom(s):
    s.b.cull()
    return s.b.aabbs, s.b.cells, s.b.indices, s.b.total


def _batch_shapes(case):
    """(grid with tile size, light count) of each view of a batch case."""
    r = random.Random(case["mix"])
    return [(r.choice(MIX), _log_int(r, case["lights_lo"], case["lights_hi"])) for _ in range(case["views"])]


def _pooled(sizes, align, dtype, width):
    """One zeroed tensor for many views, and each view's first row (rows of `width`, aligned to `align` rows)."""
    starts, at = [], 0
    for n in sizes:
        starts.append(at)
        at += -(-n // align) * align
    return torch.zeros(at, width, dtype=dtype, device="cuda"), starts


def _batch_view(ubo, lights, n, aabbs, cells, indices, total, cap=150):
    v = CfBatchView()
    v.ubo = ubo
    v.d_lights, v.d_aabbs, v.d_cells, v.d_indices, v.d_total = lights, aabbs, cells, indices, total
    v.index_capacity = ubo.sliceCountX * ubo.sliceCountY * ubo.sliceCountZ * cap
    v.light_count, v.max_lights_per_cluster = n, cap
    return v


def _prepare_batch(case, seed):
    g, r, shapes, cap = _gen(seed), random.Random(seed), _batch_shapes(case), 150
    counts = [x * y * z for (x, y, z, _), _ in shapes]
    aabbs, at_a = _pooled(counts, 8, torch.float32, 8)
    cells, at_c = _pooled(counts, 32, torch.int32, 2)
    indices, at_i = _pooled([c * cap for c in counts], 64, torch.int32, 1)
    totals = torch.zeros(len(shapes), dtype=torch.int32, device="cuda")
    lights, views = [], []
    for i, ((x, y, z, tile), n) in enumerate(shapes):
        ubo = camera.cluster_forward_ubo(FOVY, x * tile, y * tile, 0.1, 2000.0, _random_camera(r), (x, y, z))
        lights.append(_lights(g, n, "blobs"))
        views.append(_batch_view(ubo, lights[-1].data_ptr(), n, aabbs.data_ptr() + 32 * at_a[i],
                                 cells.data_ptr() + 8 * at_c[i], indices.data_ptr() + 4 * at_i[i],
                                 totals.data_ptr() + 4 * i))
    ctx = Context(0)
    batch, stream = Batch(ctx), torch.cuda.Stream()
    batch.set_views(views)
    torch.cuda.synchronize()
    batch.generate_aabbs(stream)
    stream.synchronize()
    return _State(kind="batch", ctx=ctx, batch=batch, stream=stream, lights=lights, aabbs=aabbs, cells=cells,
                  indices=indices, totals=totals)


def _run_batch(s):
    s.batch.cull(s.stream)
    return s.cells, s.indices, s.totals


def _stress_grids(case):
    return [MIX[1] if (i + case["epoch"]) % 2 == 0 else MIX[3] for i in range(case["views"])]


def _prepare_animate(case, seed):
    g, r, grids = _gen(seed), random.Random(seed), _stress_grids(case)
    n, views, cap = case["lights"], case["views"], 150
    counts = [x * y * z for x, y, z, _ in grids]
    aabbs, at_a = _pooled(counts, 8, torch.float32, 8)
    cells, at_c = _pooled(counts, 32, torch.int32, 2)
    indices, at_i = _pooled([c * cap for c in counts], 64, torch.int32, 1)
    totals = torch.zeros(views, dtype=torch.int32, device="cuda")
    centre = _blob_positions(g, n, views)
    rho, omega, phase = 1.0 + 9.0 * _u(g, views * n), 0.1 + 1.9 * _u(g, views * n), 2.0 * math.pi * _u(g, views * n)
    orbits = torch.empty(views * n, 8, device="cuda")
    orbits[:, 0], orbits[:, 1] = rho * torch.cos(phase), rho * torch.sin(phase)
    orbits[:, 2], orbits[:, 3] = torch.cos(omega / 60.0), torch.sin(omega / 60.0)
    orbits[:, 4:7], orbits[:, 7] = centre, 1.0
    pos = centre.clone()
    pos[:, 0] += orbits[:, 0]
    pos[:, 2] += orbits[:, 1]
    lights = _records(pos, _blob_radii(g, views * n), _u(g, views * n, 3))
    proj = {}
    bviews = []
    for i, (x, y, z, tile) in enumerate(grids):
        if x not in proj:
            fovy = math.radians(45.0 if case["epoch"] % 2 == 0 else 60.0)
            proj[x] = bytes(camera.cluster_forward_ubo(fovy, x * tile, y * tile, 0.1, 2000.0,
                                                       np.eye(4, dtype=np.float32), (x, y, z)))
        ubo = camera.ubo_from_bytes(proj[x])
        ubo.cameraView[:] = camera.column_major(_random_camera(r)).tolist()
        bviews.append(_batch_view(ubo, lights.data_ptr() + 48 * n * i, n, aabbs.data_ptr() + 32 * at_a[i],
                                  cells.data_ptr() + 8 * at_c[i], indices.data_ptr() + 4 * at_i[i],
                                  totals.data_ptr() + 4 * i))
    ctx = Context(0)
    batch, stream = Batch(ctx), torch.cuda.Stream()
    batch.set_views(bviews)
    torch.cuda.synchronize()
    batch.generate_aabbs(stream)
    stream.synchronize()
    return _State(kind="animate", ctx=ctx, batch=batch, stream=stream, lights=lights, orbits=orbits, aabbs=aabbs,
                  cells=cells, indices=indices, totals=totals)


def _run_animate(s):
    check(lib().cf_animate_light_orbits(s.lights.data_ptr(), s.orbits.data_ptr(), s.lights.shape[0], 1,
                                        stream_handle(s.stream)))
    s.batch.cull(s.stream)
    return s.lights, s.cells, s.indices, s.totals


def _linear_depth(case, g, r):
    w, h, near, far = case["w"], case["h"], case["near"], case["far"]
    if case["depth"] == "scatter":  # every pixel at its own depth, log-uniform over the view's range
        lin = near * torch.exp(_u(g, h, w).double() * math.log(0.9 * far / near))
    else:  # a floor, a far wall and a dozen curved objects in front
        y = ((torch.arange(h, device="cuda", dtype=torch.float64) + 0.5) / h * 2.0 - 1.0)[:, None]
        x = ((torch.arange(w, device="cuda", dtype=torch.float64) + 0.5) / w * 2.0 - 1.0)[None, :]
        wall = r.uniform(30.0, 45.0)
        lin = torch.where(y > 2.0 / wall, 2.0 / y.clamp(min=1e-3), wall + 2.0 * torch.sin(3.0 * x)).expand(h, w).clone()
        for _ in range(12):
            cx, cy, rad, d = r.uniform(-1, 1), r.uniform(-0.6, 0.9), r.uniform(0.05, 0.35), r.uniform(3.0, 28.0)
            q = 1.0 - ((x - cx) ** 2 + (y - cy) ** 2) / (rad * rad)
            lin = torch.where(q > 0, torch.minimum(lin, d - 2.0 * rad * torch.sqrt(q.clamp(min=0.0))), lin)
    z = ((near * far / lin - far) / (near - far)).clamp(0.0, 1.0 - 2.0 ** -24).float()
    z[_u(g, h, w) < 0.01] = 1.0  # some sky
    return z


def _prepare_lists(case, seed):
    g, r = _gen(seed), random.Random(seed)
    b = _Buffers(_ubo(case, _view_matrix(case, seed)), _lights(g, case["lights"], case["scene"]), case["cap"])
    b.cull()
    return g, r, b, int(b.total.item())


def _prepare_lookup(case, seed):
    g, r, b, total = _prepare_lists(case, seed)
    return _State(kind="lookup", b=b, total=total, depth=_linear_depth(case, g, r), check=case["check"])


def _run_lookup(s):
    b = s.b
    return lookup_clusters(b.ubo, s.depth, b.cells, b.indices, b.lights, s.total, b.n, b.cap, b.aabbs, s.check,
                           torch.cuda.current_stream())


def _gbuffer(case, seed):
    """(state without lists, camera position, G-buffer) of a shading case."""
    g, r, b, total = _prepare_lists(case, seed)
    z = _linear_depth(case, g, r)
    h, w = z.shape
    inv_p = torch.tensor(list(b.ubo.cameraInverseProjection), dtype=torch.float64, device="cuda").reshape(4, 4)
    inv_v = torch.linalg.inv(torch.tensor(list(b.ubo.cameraView), dtype=torch.float64).reshape(4, 4)).cuda()
    clip = torch.ones(h, w, 4, dtype=torch.float64, device="cuda")
    clip[..., 0] = (torch.arange(w, device="cuda") + 0.5) / w * 2.0 - 1.0
    clip[..., 1] = ((torch.arange(h, device="cuda") + 0.5) / h * 2.0 - 1.0)[:, None]
    clip[..., 2] = z
    v = clip @ inv_p
    world = (v / v[..., 3:4]) @ inv_v
    eye = inv_v[3, :3]
    if case["depth"] == "scatter":
        nrm = torch.randn(h, w, 3, generator=g, device="cuda", dtype=torch.float64)
    else:  # geometric normals, bent a little as by a normal map
        nrm = torch.linalg.cross(torch.gradient(world[..., :3], dim=1)[0], torch.gradient(world[..., :3], dim=0)[0])
        nrm = nrm / nrm.norm(dim=-1, keepdim=True).clamp(min=1e-30)
        nrm = nrm + 0.2 * torch.randn(h, w, 3, generator=g, device="cuda", dtype=torch.float64)
    nrm = nrm / nrm.norm(dim=-1, keepdim=True)
    nrm = torch.where(((eye - world[..., :3]) * nrm).sum(-1, keepdim=True) < 0, -nrm, nrm)
    gb = torch.empty(h, w, 12, device="cuda")
    gb[..., 0:3], gb[..., 3], gb[..., 4:7] = world[..., :3].float(), z, nrm.float()
    gb[..., 7] = _u(g, h, w)
    gb[..., 8:11] = _u(g, h, w, 3)
    gb[..., 11] = 0.05 + 0.95 * _u(g, h, w)
    return b, total, eye.tolist(), gb


def _prepare_shade(case, seed):
    b, total, eye, gb = _gbuffer(case, seed)
    return _State(kind="shade", b=b, total=total, eye=eye, pc=CfPBRPushConstant(*PC), gb=gb)


def _run_shade(s):
    b = s.b
    return shade_clusters(b.ubo, s.eye, s.pc, s.gb, b.cells, b.indices, s.total, b.lights, b.n,
                          torch.cuda.current_stream())


def _prepare_frustum(case, seed):
    g, n = _gen(seed), case["boxes"]
    centre, half = 400.0 * _u(g, n, 3) - 200.0, (0.5 + 9.5 * _u(g, n, 3)) / 2.0
    boxes = torch.zeros(n, 8, device="cuda")
    boxes[:, 0:3], boxes[:, 4:7] = centre - half, centre + half
    r = random.Random(seed)
    view = camera.look_at_rh((r.uniform(-20, 20), 10.0, 60.0), (0.0, 0.0, 0.0))
    cmds = torch.zeros(n, 4, dtype=torch.int32, device="cuda")
    cmds[:, 0], cmds[:, 1] = 36, 1
    return _State(kind="frustum", f=camera.frustum_ubo(FOVY, 16.0 / 9.0, 0.1, 500.0, view), boxes=boxes, cmds=cmds)


def _run_frustum(s):
    frustum_cull(s.f, s.boxes, s.cmds, None, torch.cuda.current_stream())
    return s.cmds


_PREPARE = {"frame": _prepare_frame, "zoom": _prepare_zoom, "batch": _prepare_batch, "animate": _prepare_animate,
            "lookup": _prepare_lookup, "shade": _prepare_shade, "frustum": _prepare_frustum}
_RUN = {"frame": _run_frame, "zoom": _run_zoom, "batch": _run_batch, "animate": _run_animate, "lookup": _run_lookup,
        "shade": _run_shade, "frustum": _run_frustum}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state.kind](state)


# ---- what a pass cannot do without --------------------------------------------


def _mean_list(lights, scene):
    """Listed lights per cluster, from what was measured on the scenes (and capped lists: less than in proportion)."""
    return 4.7 * (lights / 1024.0) ** 0.75 if scene == "box" else 13.6 * (lights / 16384.0) ** 0.75


def _cull_work(grid, lights, mean, aabbs_written=False):
    """Lights and boxes read once, cells and the list written once; a transform per light and a test per hit."""
    c = grid[0] * grid[1] * grid[2]
    hits = c * min(150.0, mean)
    return {"bytes": 48 * lights + 32 * c + 8 * c + 4 * hits + (32 * c if aabbs_written else 0),
            "flops": 22 * lights + 11 * hits}


def work(case):
    k = case["kind"]
    if k in ("frame", "zoom"):
        return _cull_work((case["x"], case["y"], case["z"]), case["lights"], _mean_list(case["lights"], case["scene"]),
                          k == "zoom")
    if k in ("batch", "animate"):
        shapes = _batch_shapes(case) if k == "batch" else [(gr, case["lights"]) for gr in _stress_grids(case)]
        # cameras of the mix look past some of the blobs: fewer listed lights than the headline view has
        parts = [_cull_work(gr[:3], n, 0.4 * _mean_list(n, "blobs")) for gr, n in shapes]
        w = {q: sum(p[q] for p in parts) for q in ("bytes", "flops")}
        if k == "animate":  # orbit state read, offset and position written
            w["bytes"] += 56 * case["views"] * case["lights"]
        return w
    if k == "frustum":
        return {"bytes": 36 * case["boxes"], "flops": 48 * case["boxes"]}
    px = case["w"] * case["h"]
    mean = min(150.0, _mean_list(case["lights"], case["scene"]))
    c = case["x"] * case["y"] * case["z"]
    lists = 48 * case["lights"] + 8 * c + 4 * c * mean
    if k == "lookup":
        return {"bytes": px * 36 + lists + 32 * c, "flops": px * (60 + 9 * mean)}
    return {"bytes": px * 64 + lists, "flops": px * (60 + 150 * mean)}


# ---- the outputs in 64 bits ----------------------------------------------------


def _exact_aabbs(case, seed):
    u = _ubo(case, _view_matrix(case, seed))
    ip = torch.tensor(list(u.cameraInverseProjection), dtype=torch.float64).reshape(4, 4)
    x, y, z = case["x"], case["y"], case["z"]

    def corner(i, j):  # a screen point unprojected, for every (j, i) of the grid
        p = torch.ones(y, x, 4, dtype=torch.float64)
        p[..., 0], p[..., 1], p[..., 2] = i[None, :] / x * 2.0 - 1.0, (j / y * 2.0 - 1.0)[:, None], 0.0
        v = p @ ip
        return v[..., :3] / v[..., 3:4]

    i, j = torch.arange(x, dtype=torch.float64), torch.arange(y, dtype=torch.float64)
    k = torch.arange(z + 1, dtype=torch.float64)
    plane = -float(u.cameraNear) * (float(u.cameraFar) / float(u.cameraNear)) ** (k / z)
    pts = []
    for c in (corner(i, j), corner(i + 1, j + 1)):
        ray = c / c[..., 2:3]
        pts += [ray[None] * plane[:-1, None, None, None], ray[None] * plane[1:, None, None, None]]
    p = torch.stack(pts)
    out = torch.zeros(z, y, x, 8, dtype=torch.float64)
    out[..., 0:3], out[..., 4:7] = p.amin(0), p.amax(0)
    return out.reshape(-1, 8)


def _exact_shade(case, seed):
    """Every light of the scene against every texel: a light outside a cluster's list is out of the texel's reach
    and adds nothing, as long as no list is capped."""
    b, _, eye, gb = _gbuffer(case, seed)
    if int(b.cells[:, 1].max()) >= case["cap"] or case["w"] * case["h"] * case["lights"] > 2.5e9:
        return None
    t = gb.reshape(-1, 12)
    intensity, base, _, falloff, mult = (float(np.float32(v)) for v in PC)
    L = b.lights.double()
    out = torch.empty(t.shape[0], 4, dtype=torch.float64, device="cuda")
    at = torch.tensor([float(np.float32(v)) for v in eye], dtype=torch.float64, device="cuda")
    for lo in range(0, t.shape[0], 65536):
        q = t[lo:lo + 65536].double()
        P, N, met, alb, rough = q[:, 0:3], q[:, 4:7], q[:, 7:8], q[:, 8:11], q[:, 11]
        V = at - P
        V = V / V.norm(dim=-1, keepdim=True)
        nov = (N * V).sum(-1).clamp(min=0.0)
        F0 = base * (1.0 - met) + alb * met
        ar = (rough + 1.0) ** 2 / 8.0
        a2 = rough ** 4
        inside = q[:, 3] < 1.0
        acc = alb * mult
        # only the pairs in reach: a distance below the light's radius
        d2 = torch.cdist(P, L[:, 0:3], compute_mode="donot_use_mm_for_euclid_dist")
        ti, li = ((d2 < L[None, :, 8]) & inside[:, None]).nonzero(as_tuple=True)
        d = L[li, 0:3] - P[ti]
        dist = d.norm(dim=-1)
        Ld = d / dist[:, None]
        H = V[ti] + Ld
        H = H / H.norm(dim=-1, keepdim=True)
        noh, nol = (N[ti] * H).sum(-1).clamp(min=0.0), (N[ti] * Ld).sum(-1).clamp(min=0.0)
        hov = (H * V[ti]).sum(-1).clamp(min=0.0)
        att = (1.0 - dist / L[li, 8]).clamp(min=0.0) / dist ** falloff
        rad = L[li, 4:7] * (att * intensity)[:, None]
        den = noh * noh * (a2[ti] - 1.0) + 1.0
        D = a2[ti] / (math.pi * den * den)
        k = ar[ti]
        G = nol / (nol * (1.0 - k) + k) * (nov[ti] / (nov[ti] * (1.0 - k) + k))
        F = F0[ti] + (1.0 - F0[ti]) * ((1.0 - hov).clamp(0.0, 1.0) ** 5)[:, None]
        spec = F * (D * G / (4.0 * nov[ti] * nol + 0.0001))[:, None]
        diff = (1.0 - F) * (1.0 - met[ti]) * alb[ti] / math.pi
        acc.index_add_(0, ti, (diff + spec) * rad * nol[:, None])
        out[lo:lo + 65536, 0:3], out[lo:lo + 65536, 3] = acc, inside.double()
    return out.reshape(gb.shape[0], gb.shape[1], 4)


def _exact_animate(case, seed):
    s = _prepare_animate(case, seed)
    lights, o = s.lights.double(), s.orbits.double()
    lights[:, 0] = o[:, 4] + (o[:, 2] * o[:, 0] - o[:, 3] * o[:, 1])
    lights[:, 1] = o[:, 5]
    lights[:, 2] = o[:, 6] + (o[:, 3] * o[:, 0] + o[:, 2] * o[:, 1])
    lights[:, 3] = o[:, 7]
    return lights


def exact(case, seed):
    """Cells, lists, counters and lookup records are whole numbers and bytes; what is computed in floats is here."""
    if case["kind"] == "zoom":
        return _exact_aabbs(case, seed), None, None, None
    if case["kind"] == "animate":
        return _exact_animate(case, seed), None, None, None
    if case["kind"] == "shade":
        return _exact_shade(case, seed)
    return None
