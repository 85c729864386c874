"""Performance cases of the ray-tracing core: what a program that uses it does,
through its public entry points (the rtcore binding of the C ABI), from one
small query to whole path-traced frames.

A case is a dict of plain values; "op" names the call:

  frame    rt_trace_rays: the sample's pipeline (raygen, traversal of a
           two-level structure, closest-hit / miss programs) into an RGBA32F image
  rays     rt_trace_closest / rt_trace_any over a device ray buffer
  build    rt_build_blas of one geometry
  refit    rt_refit_blas after every vertex moved
  pt       rt_path_trace: a progressive frame
  learned  rt_path_trace_cached: a frame whose paths end in the MLP cache,
           which trains on the frame's own path tails
  batch    rt_batch_launch of a plan recorded once: several scenes of uneven
           triangle counts and resolutions
  query    rt_cache_query: MLP cache inference
  train    rt_cache_train: Adam steps on path-tail samples

Scenes are the repository's seeded generators: the triangle soup, the box with
icospheres, and the sample's quads under two instances.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "build-up-phase_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import rtcore  # noqa: E402
import rtcore.batch as batch  # noqa: E402
import rtcore.scenes as scenes  # noqa: E402

_context = None


def context():
    """One context for the whole program, as its users hold it."""
    global _context
    if _context is None:
        _context = rtcore.Context(0)
    return _context


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # The sample itself: one 1200x800 frame of its two instances of two quads.
        {"name": "frame_sample", "op": "frame", "width": 1200, "height": 800},
        # A handful of visibility probes in a small scene (picking, audio or AI
        # line-of-sight queries each tick): the call's latency counts.
        {"name": "probes_small", "op": "rays", "kind": "any", "tris": 20000, "instances": 0, "primary_w": 0,
         "primary_h": 0, "incoherent": 4097},
        # The ray-casting workload: 1M-triangle soup, 1920x1080 primary rays and
        # as many incoherent ones in one call.
        {"name": "rays_soup_1m", "op": "rays", "kind": "closest", "tris": 1000000, "instances": 0,
         "primary_w": 1920, "primary_h": 1080, "incoherent": 1920 * 1080},
        # An instanced scene: closest hits through a top-level structure of 64
        # rotated, scaled instances of three meshes.
        {"name": "rays_instances", "op": "rays", "kind": "closest", "tris": 60000, "instances": 64,
         "primary_w": 641, "primary_h": 479, "incoherent": 500003},
        # A small mesh loaded or changed at run time.
        {"name": "build_small", "op": "build", "scene": "soup", "tris": 12345, "morton30": False},
        # The 1M-triangle soup's build.
        {"name": "build_soup_1m", "op": "build", "scene": "soup", "tris": 1000000, "morton30": False},
        # Animated geometry: the 2M-triangle box refitted each frame.
        {"name": "refit_box_2m", "op": "refit", "spheres": 40, "freq": 50},
        # A path-traced 1920x1080 frame of the 2M-triangle box, four samples.
        {"name": "pt_box_2m", "op": "pt", "spheres": 40, "freq": 50, "width": 1920, "height": 1080, "spp": 4,
         "depth": 8},
        # The learned form: the 8M-triangle box, 65,536 training paths per
        # sample in Adam batches of 4,096, four samples.
        {"name": "learned_box_8m", "op": "learned", "spheres": 160, "freq": 50, "width": 1920, "height": 1080,
         "spp": 4, "depth": 8, "train_paths": 65536, "train_batch": 4096},
        # Several small scenes of uneven sizes in one recorded launch.
        {"name": "batch_small", "op": "batch", "scenes": 6, "min_tris": 10000, "max_tris": 200000, "res": 320,
         "spp": 2, "depth": 8},
        # Cache inference for every pixel of a 1920x1080 frame.
        {"name": "query_2m", "op": "query", "n": 1920 * 1080},
        # Online training on one frame's 65,536 path tails, batches of 4,096.
        {"name": "train_64k", "op": "train", "n": 65536, "batch": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["frame", "rays", "rays", "build", "build", "refit", "pt", "learned", "batch", "query", "train"])
    if op == "frame":
        return {"op": op, "width": _log(rng, 33, 2048), "height": _log(rng, 33, 1600)}
    if op == "rays":
        w = rng.choice([0, _log(rng, 8, 1920)])
        return {"op": op, "kind": rng.choice(["closest", "any"]), "tris": _log(rng, 300, 1000000),
                "instances": rng.choice([0, 0, _log(rng, 2, 300)]), "primary_w": w,
                "primary_h": _log(rng, 8, 1080) if w else 0, "incoherent": _log(rng, 33, 2000000)}
    if op == "build":
        return {"op": op, "scene": rng.choice(["soup", "box"]), "tris": _log(rng, 1000, 2000000),
                "morton30": rng.random() < 0.25}
    if op == "refit":
        return {"op": op, "spheres": rng.randint(1, 40), "freq": _log(rng, 4, 50)}
    if op == "pt":
        return {"op": op, "spheres": rng.randint(1, 40), "freq": _log(rng, 4, 50), "width": _log(rng, 65, 1920),
                "height": _log(rng, 49, 1080), "spp": rng.randint(1, 4), "depth": rng.randint(2, 8)}
    if op == "learned":
        return {"op": op, "spheres": rng.randint(1, 40), "freq": _log(rng, 4, 50), "width": _log(rng, 320, 1280),
                "height": _log(rng, 200, 720), "spp": rng.randint(1, 4), "depth": 8,
                "train_paths": _log(rng, 4096, 65536), "train_batch": rng.choice([4096, 8192, 16384])}
    if op == "batch":
        return {"op": op, "scenes": rng.randint(2, 12), "min_tris": 10000, "max_tris": 300000,
                "res": _log(rng, 64, 512), "spp": rng.randint(1, 2), "depth": 8}
    if op == "query":
        return {"op": op, "n": _log(rng, 100, 1920 * 1080)}
    return {"op": op, "n": _log(rng, 1000, 65536), "batch": rng.choice([4096, 8192, 16384])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _gpu(a):
    """A numpy array's bytes on the GPU."""
    return torch.from_numpy(np.ascontiguousarray(a).reshape(-1).view(np.uint8)).cuda()


def _zeros(nbytes):
    return torch.zeros(max(1, int(nbytes)), dtype=torch.uint8, device="cuda")


def _empty(nbytes):
    return torch.empty(max(1, int(nbytes)), dtype=torch.uint8, device="cuda")


def _geometry(dv, n_vertices, di, n_tris, transform=None):
    g = rtcore.GeometryTriangles()
    g.vertices, g.vertex_stride, g.max_vertex = dv.data_ptr(), 12, n_vertices - 1
    g.index_type, g.indices, g.tri_count, g.flags = rtcore.RT_INDEX_UINT32, di.data_ptr(), n_tris, 1
    if transform is not None:
        g.transform = transform.data_ptr()
    return g


class Mesh:
    """Geometry on the device with the structure and scratch it is built into."""

    def __init__(self, v, i, flags=0, build=True):
        ctx = context()
        self.dv, self.di, self.n_vertices, self.n_tris, self.flags = _gpu(v), _gpu(i), len(v), len(i), flags
        self.geoms = [_geometry(self.dv, len(v), self.di, len(i))]
        self.sizes = ctx.blas_sizes([len(i)], flags)
        self.accel = _zeros(self.sizes.accel_bytes)
        if build:
            scratch = _empty(self.sizes.scratch_bytes)
            self.build(scratch)
            ctx.sync()

    def build(self, scratch):
        context().build_blas(self.geoms, self.flags, self.accel, self.sizes.accel_bytes, scratch,
                             self.sizes.scratch_bytes)


def _rotation(rng):
    q = rng.normal(size=4)
    w, x, y, z = q / np.linalg.norm(q)
    return np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                     [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                     [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]])


def _tlas(inst):
    ctx = context()
    d = _gpu(inst)
    sz = ctx.tlas_sizes(len(inst))
    accel, scratch = _zeros(sz.accel_bytes), _empty(sz.scratch_bytes)
    ctx.build_tlas(d, len(inst), 0, accel, sz.accel_bytes, scratch, sz.scratch_bytes)
    ctx.sync()
    return accel


def _sample_inputs(seed):
    """The sample's quads, instances, record colours and camera, each a little
    moved by the seed (an animated camera and objects)."""
    rng = np.random.default_rng(seed)
    inst_t = scenes.REF8_INSTANCE_TRANSFORMS.copy()
    inst_t[:, :, 3] += rng.uniform(-0.2, 0.2, (2, 3)).astype(np.float32)
    colors = rng.uniform(0.05, 0.95, (4, 3)).astype(np.float32)
    pos = np.array([0.0, 0.0, 10.0], np.float32) + rng.uniform(-0.3, 0.3, 3).astype(np.float32)
    return inst_t, colors, pos, float(np.float32(60.0))


def _box_mesh_shape(tris):
    spheres = max(1, min(200, tris // 25000))
    return spheres, max(1, int(round(math.sqrt(max(tris - 14, 20) / (20.0 * spheres)))))


def _mesh_arrays(scene, tris, seed):
    if scene == "soup":
        return scenes.soup(seed, tris)
    return scenes.box(seed, *_box_mesh_shape(tris))[:2]


def _primary(case, lo, hi):
    """Primary rays of a camera in front of the box [lo, hi], made on the GPU."""
    w, h = case["primary_w"], case["primary_h"]
    if w * h == 0:
        return None
    c = (lo + hi) * 0.5
    cam = rtcore.Camera((float(c[0]), float(c[1]), float(hi[2] + 1.5 * (hi[0] - lo[0]))), 60.0)
    out = _empty(w * h * 32)
    context().generate_primary_rays(cam, w, h, 0.0, 1e30, out)
    return out


def _instance_seeds(seed):
    return [seed * 3 + k for k in range(3)]


def _instance_table(case, seed):
    rng = np.random.default_rng(seed)
    n = case["instances"]
    inst = np.zeros(n, scenes.INSTANCE_DTYPE)
    side = max(1, int(math.ceil(n ** (1 / 3))))
    for k in range(n):
        cell = np.array([k % side, (k // side) % side, k // (side * side)], np.float64)
        inst[k]["transform"][:, :3] = _rotation(rng) * rng.uniform(0.5, 1.1)
        inst[k]["transform"][:, 3] = cell + rng.uniform(-0.2, 0.2, 3)
        inst[k]["custom_index_and_mask"] = rtcore.pack_custom_mask(k, 0xFF)
        inst[k]["sbt_offset_and_flags"] = rtcore.pack_sbt_flags(0, 1)
    return inst, float(side)


def _cache_rows(n, seed):
    """Cache inputs as a path tracer makes them: points in the box, unit
    directions and normals, albedos."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.empty(n, 12, dtype=torch.float32, device="cuda")
    x[:, 0:3] = torch.rand(n, 3, device="cuda", generator=g) * 2 - 1
    for k in (3, 6):
        d = torch.randn(n, 3, device="cuda", generator=g)
        x[:, k:k + 3] = d / d.norm(dim=1, keepdim=True).clamp_min(1e-6)
    x[:, 9:12] = torch.rand(n, 3, device="cuda", generator=g) * 0.8 + 0.1
    return x


def _cache_targets(x, seed):
    """Outgoing radiance of a smooth lighting of the box, with the noise that
    single path tails have."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 1)
    light = 1.5 + torch.sin(3.0 * x[:, 0:1]) * torch.cos(2.0 * x[:, 1:2]) + 0.5 * x[:, 7:8]
    noise = -torch.log(torch.rand(len(x), 3, device="cuda", generator=g).clamp_min(1e-6))
    t = torch.zeros(len(x), 4, dtype=torch.float32, device="cuda")
    t[:, :3] = x[:, 9:12] * light * noise
    return t


_LAYERS = [(96, 64)] + [(64, 64)] * 4 + [(64, 8)]  # padded inputs, outputs
_USED_IN, _USED_OUT = 81, 3


def _cache_params(seed):
    """He-uniform weights and small biases in the padded parameter layout."""
    rng = np.random.default_rng(seed + 2)
    parts = []
    for k, (i, o) in enumerate(_LAYERS):
        w, b = np.zeros((o, i), np.float32), np.zeros(o, np.float32)
        ui, uo = (_USED_IN if k == 0 else i), (_USED_OUT if k == 5 else o)
        w[:uo, :ui] = rng.uniform(-1, 1, (uo, ui)) * math.sqrt(6.0 / ui)
        b[:uo] = rng.uniform(-0.05, 0.05, uo)
        parts += [w.reshape(-1), b]
    return np.concatenate(parts)


def _cache(seed):
    ctx = context()
    cache = _zeros(ctx.cache_bytes())
    ctx.cache_init(cache, rtcore.cache_config(seed=seed & 0x7FFFFFFF))
    ctx.cache_set_params(cache, torch.from_numpy(_cache_params(seed)).cuda())
    ctx.sync()
    return cache


def _pt_scene(case, seed):
    """The box workload on the device: mesh, materials, lights."""
    v, i, tm, m = scenes.box(seed, case["spheres"], case["freq"])
    lights = scenes.emissive_lights(v, i, tm, m)
    mesh = Mesh(v, i)
    keep = [_gpu(tm), _gpu(m), _gpu(lights)]
    scene = rtcore.PtScene(context().address(mesh.accel), keep[0].data_ptr(), keep[1].data_ptr(), len(m),
                           keep[2].data_ptr(), len(lights))
    return mesh, keep, scene


def prepare(case, seed):
    ctx = context()
    op = case["op"]
    s = {"op": op}
    if op == "frame":
        inst_t, colors, pos, fov = _sample_inputs(seed)
        dv, di = _gpu(scenes.REF8_VERTICES), _gpu(scenes.REF8_INDICES)
        xf = [_gpu(t) for t in scenes.REF8_GEOM_TRANSFORMS]
        geoms = [_geometry(dv, 4, di, 2, t) for t in xf]
        sz = ctx.blas_sizes([2, 2])
        blas, scratch = _zeros(sz.accel_bytes), _empty(sz.scratch_bytes)
        ctx.build_blas(geoms, 0, blas, sz.accel_bytes, scratch, sz.scratch_bytes)
        inst = np.zeros(2, scenes.INSTANCE_DTYPE)
        for k in range(2):
            inst[k]["transform"] = inst_t[k]
            inst[k]["custom_index_and_mask"] = rtcore.pack_custom_mask(scenes.REF8_CUSTOM_INDEX, 0xFF)
            inst[k]["sbt_offset_and_flags"] = rtcore.pack_sbt_flags(scenes.REF8_SBT_OFFSETS[k], 1)
            inst[k]["accel_ref"] = ctx.address(blas)
        s["blas"], s["tlas"], s["colors"] = blas, _tlas(inst), _gpu(colors)
        s["sbt"] = rtcore.Sbt(s["colors"].data_ptr(), 4, 3)
        s["pipeline"] = rtcore.sample_pipeline()
        s["camera"] = rtcore.Camera(tuple(float(x) for x in pos), fov)
        s["w"], s["h"] = case["width"], case["height"]
        s["image"] = torch.zeros(s["h"], s["w"], 4, dtype=torch.float32, device="cuda")
    elif op == "rays":
        n_inst = case["instances"]
        if n_inst:
            meshes = [Mesh(*scenes.soup(sd, max(1, case["tris"] // 3))) for sd in _instance_seeds(seed)]
            inst, side = _instance_table(case, seed)
            for k in range(n_inst):
                inst[k]["accel_ref"] = ctx.address(meshes[k % 3].accel)
            s["keep"], s["accel"] = meshes, _tlas(inst)
            lo, hi = np.full(3, -0.5, np.float32), np.full(3, side, np.float32)
        else:
            mesh = Mesh(*scenes.soup(seed, case["tris"]))
            s["keep"], s["accel"] = mesh, mesh.accel
            lo, hi = np.zeros(3, np.float32), np.ones(3, np.float32)
        # a shadow ray stops at its light, a closest-hit ray goes on
        tmax = 0.25 if case["kind"] == "any" else 1e30
        parts = [_primary(case, lo, hi), _gpu(scenes.incoherent_rays(seed + 5, case["incoherent"], lo, hi, tmax))]
        s["rays"] = torch.cat([p for p in parts if p is not None])
        s["n"] = s["rays"].numel() // 32
        s["addr"] = ctx.address(s["accel"])
        s["any"] = case["kind"] == "any"
        if s["any"]:
            s["occluded"] = _zeros(s["n"])
        else:
            s["hits"] = _zeros(s["n"] * 16)
            f, i = s["hits"].view(torch.float32).view(-1, 4), s["hits"].view(torch.int32).view(-1, 4)
            s["out"] = {"t": f[:, 0], "uv": f[:, 2:4], "prim": i[:, 1]}
    elif op == "build":
        v, i = _mesh_arrays(case["scene"], case["tris"], seed)
        flags = rtcore.RT_BUILD_MORTON30 if case["morton30"] else 0
        s["mesh"] = Mesh(v, i, flags, build=False)
        s["scratch"] = _empty(s["mesh"].sizes.scratch_bytes)
    elif op == "refit":
        v, i = scenes.box(seed, case["spheres"], case["freq"])[:2]
        s["mesh"] = Mesh(v, i)
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        p = s["mesh"].dv.view(torch.float32).view(-1, 3)
        a = torch.rand(3, device="cuda", generator=g)
        s["moved"] = (p + 0.01 * torch.sin(7.0 * p[:, [1, 2, 0]] + 6.0 * a)).contiguous()
        s["geoms"] = [_geometry(s["moved"], len(v), s["mesh"].di, len(i))]
        s["bytes"] = rtcore.refit_scratch_bytes(len(i))
        s["scratch"] = _empty(s["bytes"])
    elif op in ("pt", "learned"):
        s["mesh"], s["keep"], s["scene"] = _pt_scene(case, seed)
        w, h = case["width"], case["height"]
        s["params"] = rtcore.PtParams(rtcore.Camera(*scenes.BOX_CAMERA), w, h, case["spp"], 0, case["depth"], 3,
                                      seed, 1e-4, 0)
        s["accum"] = torch.zeros(h, w, 4, dtype=torch.float32, device="cuda")
        if op == "learned":
            s["checkpoint"] = _cache(seed)
            s["cache"] = s["checkpoint"].clone()
            s["cp"] = rtcore.PtCacheParams(s["cache"].data_ptr(), case["train_paths"], case["train_batch"])
            s["weights"] = torch.zeros(rtcore.load().rt_cache_param_count(), dtype=torch.float32, device="cuda")
            s["bytes"] = ctx.pt_cached_scratch_bytes(s["params"], s["cp"])
        else:
            s["bytes"] = ctx.pt_scratch_bytes(s["params"])
        s["scratch"] = _empty(s["bytes"])
    elif op == "batch":
        specs = batch.batch_specs(case["scenes"], case["min_tris"], case["max_tris"], seed)
        for k, sp in enumerate(specs):  # resolutions by place: a program's targets stay as its scenes change
            sp.width = (case["res"], case["res"] // 2 + 1, 2 * case["res"] // 3)[k % 3]
            sp.height = max(1, sp.width * 3 // 4)
        s["scenes"] = [batch.GpuScene(ctx, sp, batch.host_scene(sp)) for sp in specs]
        p = batch.batch_params(case["spp"], case["depth"], seed)
        table = [sc.batch_scene() for sc in s["scenes"]]
        nb = ctx.batch_scratch_bytes(table, p)
        s["scratch"] = _empty(nb)
        s["plan"] = ctx.batch_plan(table, p, s["scratch"], nb, graph=True)
        s["images"] = [sc.accum for sc in s["scenes"]]
    else:
        x = _cache_rows(case["n"], seed)
        s["inputs"], s["n"] = x, case["n"]
        if op == "query":
            s["cache"] = _cache(seed)
            s["out"] = torch.zeros(case["n"], 4, dtype=torch.float32, device="cuda")
        else:
            s["checkpoint"], s["targets"], s["batch"] = _cache(seed), _cache_targets(x, seed), case["batch"]
            s["cache"] = s["checkpoint"].clone()
            s["weights"] = torch.zeros(rtcore.load().rt_cache_param_count(), dtype=torch.float32, device="cuda")
            s["loss"] = torch.zeros(1, dtype=torch.float32, device="cuda")
    ctx.sync()
    return s


def run(s):
    ctx = context()
    op = s["op"]
    if op == "frame":
        ctx.trace_rays(s["pipeline"], s["sbt"], ctx.address(s["tlas"]), s["camera"], s["image"], s["w"], s["h"])
        return s["image"]
    if op == "rays":
        if s["any"]:
            ctx.trace_any(s["addr"], s["rays"], s["occluded"], s["n"])
            return s["occluded"]
        ctx.trace_closest(s["addr"], s["rays"], s["hits"], s["n"])
        return s["out"]
    if op == "build":
        s["mesh"].build(s["scratch"])
        return s["mesh"].accel
    if op == "refit":
        m = s["mesh"]
        ctx.refit_blas(s["geoms"], m.accel, m.sizes.accel_bytes, s["scratch"], s["bytes"])
        return m.accel
    if op == "pt":
        ctx.path_trace(s["scene"], s["params"], s["accum"], s["scratch"], s["bytes"])
        return s["accum"]
    if op == "learned":
        # every frame starts from the saved checkpoint (a shot rendered frame by frame)
        s["cache"].copy_(s["checkpoint"])
        ctx.path_trace_cached(s["scene"], s["params"], s["cp"], s["accum"], s["scratch"], s["bytes"])
        ctx.cache_get_params(s["cache"], s["weights"])
        return {"image": s["accum"], "weights": s["weights"]}
    if op == "batch":
        s["plan"].launch(0)
        return s["images"]
    if op == "query":
        ctx.cache_query(s["cache"], s["inputs"], s["out"], s["n"])
        return s["out"]
    s["cache"].copy_(s["checkpoint"])
    ctx.cache_train(s["cache"], s["inputs"], s["targets"], s["n"], s["batch"], s["loss"])
    ctx.cache_get_params(s["cache"], s["weights"])
    return {"weights": s["weights"], "loss": s["loss"]}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

# A built structure's bytes per triangle: its 48-byte record and, at about 0.28
# wide nodes of 80 bytes per triangle, its nodes.
_ACCEL_BYTES = 48 + 23
_PARAMS = sum(i * o + o for i, o in _LAYERS)
_QUERY_FLOPS = 2 * (81 * 64 + 4 * 64 * 64 + 64 * 3)


def work(case):
    op = case["op"]
    if op == "frame":
        return {"bytes": 16 * case["width"] * case["height"], "flops": 0}
    if op == "rays":
        n = case["primary_w"] * case["primary_h"] + case["incoherent"]
        return {"bytes": n * (32 + (1 if case["kind"] == "any" else 16)) + case["tris"] * _ACCEL_BYTES, "flops": 0}
    if op == "build":
        return {"bytes": case["tris"] * (12 + 36 + _ACCEL_BYTES), "flops": 0}
    if op == "refit":
        # vertices (about half as many as triangles) and indices in, the
        # records' ids and the nodes' child data in, records and nodes out
        n = 20 * case["freq"] ** 2 * case["spheres"] + 14
        return {"bytes": n * (6 + 12 + 12 + 48 + 23 + 23), "flops": 0}
    if op in ("pt", "learned"):
        n = 20 * case["freq"] ** 2 * case["spheres"] + 14
        b = 32 * case["width"] * case["height"] + n * _ACCEL_BYTES
        if op == "pt":
            return {"bytes": b, "flops": 0}
        rows = case["width"] * case["height"] * case["spp"]
        return {"bytes": b + 16 * _PARAMS,
                "flops": rows * _QUERY_FLOPS + 3 * case["spp"] * case["train_paths"] * _QUERY_FLOPS}
    if op == "batch":
        tris = math.sqrt(case["min_tris"] * case["max_tris"])
        return {"bytes": case["scenes"] * (32 * case["res"] ** 2 * 0.43 + tris * _ACCEL_BYTES), "flops": 0}
    if op == "query":
        return {"bytes": 64 * case["n"] + 2 * _PARAMS, "flops": case["n"] * _QUERY_FLOPS}
    return {"bytes": 64 * case["n"] + 2 * 12 * _PARAMS, "flops": 3 * case["n"] * _QUERY_FLOPS}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def _exact_frame(case, seed):
    """The sample's image from its eight triangles, every ray against each."""
    inst_t, colors, pos, fov = _sample_inputs(seed)
    w, h = case["width"], case["height"]
    dev = "cuda"
    f64 = torch.float64
    ay = math.tan(math.radians(fov) * 0.5)
    ax = ay * w / h
    x = ((torch.arange(w, device=dev, dtype=f64) + 0.5) / w * 2 - 1) * ax
    y = -((torch.arange(h, device=dev, dtype=f64) + 0.5) / h * 2 - 1) * ay
    d = torch.stack([x[None, :].expand(h, w), y[:, None].expand(h, w), torch.full((h, w), -1.0, device=dev, dtype=f64)], -1)
    o = torch.tensor(pos.astype(np.float64), device=dev)
    best = torch.full((h, w), math.inf, device=dev, dtype=f64)
    img = torch.zeros(h, w, 4, device=dev, dtype=f64)
    img[..., 2] = float(np.float32(0.2))
    for k in range(2):
        for g in range(2):
            for p in range(2):
                v = scenes.REF8_VERTICES[scenes.REF8_INDICES[p]].astype(np.float64)
                for m in (scenes.REF8_GEOM_TRANSFORMS[g], inst_t[k]):
                    v = v @ m[:, :3].astype(np.float64).T + m[:, 3].astype(np.float64)
                v = torch.tensor(v, device=dev)
                e1, e2 = v[1] - v[0], v[2] - v[0]
                q = torch.linalg.cross(d, e2.expand_as(d))
                det = q @ e1
                s = o - v[0]
                r = torch.linalg.cross(s, e1)
                bu, bv, t = (q @ s) / det, (d @ r) / det, (e2 @ r) / det
                hit = (bu >= 0) & (bv >= 0) & (bu + bv <= 1) & (t >= 0) & (t <= 100) & (t < best)
                c = torch.empty(h, w, 4, device=dev, dtype=f64)
                c[..., 3] = 0
                if k == 1 and g == 1 and p == 1:
                    c[..., 0], c[..., 1], c[..., 2] = 1 - bu - bv, bu, bv
                else:
                    c[..., :3] = torch.tensor(colors[scenes.REF8_SBT_OFFSETS[k] + g].astype(np.float64), device=dev)
                img = torch.where(hit[..., None], c, img)
                best = torch.where(hit, t, best)
    return img


def _encode(x):
    pn = (x[:, 0:3].double() + 1.0) / 2.0
    cols = []
    for a in range(3):
        for k in range(12):
            arg = math.pi * (2 ** k) * pn[:, a]
            cols += [torch.sin(arg), torch.cos(arg)]
    return torch.cat([torch.stack(cols, 1), x[:, 3:12].double()], 1)


def _weights(p):
    out, o = [], 0
    for i, n in _LAYERS:
        out.append((p[o:o + n * i].view(n, i), p[o + n * i:o + n * i + n]))
        o += n * i + n
    return out


def _network(p, x):
    a = torch.nn.functional.pad(_encode(x), (0, 96 - _USED_IN))
    layers = _weights(p)
    for w, b in layers[:-1]:
        a = torch.relu(a @ w.t() + b)
    w, b = layers[-1]
    return (a @ w.t() + b)[:, :_USED_OUT]


def exact(case, seed):
    op = case["op"]
    if op == "frame":
        return _exact_frame(case, seed)
    if op not in ("query", "train"):
        # hits, images and structures: an independent 64-bit answer would take
        # every ray against every triangle (minutes); images depend on the
        # random streams as well
        return None
    x = _cache_rows(case["n"], seed)
    p = torch.from_numpy(_cache_params(seed)).cuda().double()
    if op == "query":
        y = torch.cat([_network(p, c) for c in x.split(1 << 18)])
        return torch.nn.functional.pad(y, (0, 1))
    t = _cache_targets(x, seed)[:, :3].double()
    m, v, loss = torch.zeros_like(p), torch.zeros_like(p), None
    for step, k in enumerate(range(0, case["n"], case["batch"]), 1):
        q = p.clone().requires_grad_()
        y = _network(q, x[k:k + case["batch"]])
        loss = ((y - t[k:k + case["batch"]]) ** 2 / (y.detach() ** 2 + 0.01)).mean()
        g, = torch.autograd.grad(loss, q)
        m, v = 0.9 * m + 0.1 * g, 0.99 * v + 0.01 * g * g
        p = p - 1e-3 * (m / (1 - 0.9 ** step)) / (torch.sqrt(v / (1 - 0.99 ** step)) + 1e-8)
    return {"weights": p, "loss": loss.detach().reshape(1)}
