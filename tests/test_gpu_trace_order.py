"""Hits that depend on the order of the tests unless the traversal sees to it:
coincident triangles, and rays that start on them, so that where a box lets the
ray in and another triangle's distance differ by rounding alone.  The kernels
test records in batches; the answers have to be the oracle's, which tests them
node by node, and the same each time -- in every kernel: one level, instances,
the path tracer's launches over two queues, and those over several scenes."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import GpuBlas, GpuTlas, dev, gpu_trace_closest, host, ptr_of

pytestmark = pytest.mark.gpu

N = 1_000_000


def _walls(seed, walls=60, copies=12, flat=True):
    """Triangles, axis-parallel or not, each with copies on it, a rounding error
    off it along one axis and (even seeds) beside it."""
    rng = np.random.default_rng(seed)
    tris = []
    for _ in range(walls):
        axis = rng.integers(3)
        centre, t = rng.uniform(-1, 1, 3), rng.uniform(-2, 2, (3, 3))
        if flat:
            t[:, axis] = 0
        for k in range(copies):
            c = t + centre
            if k % 3 == 1:
                c[:, axis] += rng.normal(0, 1e-7)
            if k % 3 == 2:
                c += rng.normal(0, 1e-6, (1, 3)) * (seed % 2 == 0)
            tris.append(c)
    order = rng.permutation(len(tris)).astype(np.uint32)
    return (np.array(tris, np.float32).reshape(-1, 3),
            (3 * order[:, None] + np.arange(3, dtype=np.uint32)).astype(np.uint32), None)


def _rays_from(item, seed, n=N):
    """Rays that start on the triangles, as rounding leaves a point on them."""
    import rtcore.scenes as S
    v, i, _ = item
    rng = np.random.default_rng(seed)
    w = rng.dirichlet((1, 1, 1), n)
    p = (v[i[rng.integers(len(i), size=n)]].astype(np.float64) * w[:, :, None]).sum(1)
    d = rng.normal(size=(n, 3))
    rays = np.zeros(n, S.RAY_DTYPE)
    rays["org"], rays["dir"], rays["tmax"] = p, d / np.linalg.norm(d, axis=1)[:, None], 1e30
    return rays


def _instances(turned):
    from oracle import INSTANCE_DTYPE
    inst = np.zeros(1, INSTANCE_DTYPE)
    inst["transform"] = np.eye(4, dtype=np.float32)[:3]
    if turned:
        c, s = np.cos(0.3), np.sin(0.3)
        inst["transform"][0, :, :3] = [[c, -s, 0], [s, c, 0], [0, 0, 1]]
    inst["custom_index_and_mask"] = 0xFF << 24
    return inst


@pytest.mark.parametrize("flat", [True, False])
@pytest.mark.parametrize("seed", [12, 14, 15, 16])
def test_rays_from_coincident_triangles_match_oracle(ctx, orc, seed, flat):
    item = _walls(seed, flat=flat)
    rays = _rays_from(item, seed)
    g = GpuBlas(ctx, [item])
    ob, rc = orc.build_blas([item])
    assert rc == 0
    ho = orc.trace_closest(ob, rays)[0]
    for _ in range(2):
        assert gpu_trace_closest(ctx, g.addr, rays).tobytes() == ho.tobytes()
    for turned in (False, True):
        inst = _instances(turned)
        inst["accel_ref"] = [g.addr]
        gt = GpuTlas(ctx, inst)
        inst["accel_ref"] = [ptr_of(ob)]
        ot, rc = orc.build_tlas(inst)
        assert rc == 0
        hg, xg = gpu_trace_closest(ctx, gt.addr, rays, ext=True)
        ho, _, xo = orc.trace_closest(ot, rays, ext=True)
        assert hg.tobytes() == ho.tobytes(), turned
        assert xg.tobytes() == xo.tobytes(), turned


def _box_of_walls(seed):
    """A closed box around coincident walls, every triangle of its own colour,
    some of the box's emitting."""
    import rtcore.scenes as S
    v, i, _ = _walls(seed, walls=40)
    bv, bi = S.box(seed, 0, 1)[:2]
    i = np.concatenate([i, bi + len(v)]).astype(np.uint32)
    v = np.concatenate([v * np.float32(0.3), bv]).astype(np.float32)
    m = np.zeros(len(i), S.MATERIAL_DTYPE)
    m["albedo"] = np.random.default_rng(seed).uniform(0.3, 0.9, (len(i), 3))
    m["emission"][-len(bi)::3] = 2.0
    return v, i, np.arange(len(i), dtype=np.uint32), m


def test_coincident_walls_path_traced_match_oracle(ctx, orc):
    import rtcore
    import rtcore.scenes as S
    import torch
    w, h, spp, depth, seed = 320, 200, 8, 8, 0x5EED0003
    v, i, tm, m = _box_of_walls(20)
    lights = S.emissive_lights(v, i, tm, m)
    blas = GpuBlas(ctx, [(v, i, None)])
    keep = [dev(tm), dev(m), dev(lights)]
    sc = rtcore.PtScene(blas.addr, keep[0].data_ptr(), keep[1].data_ptr(), len(m), keep[2].data_ptr(), len(lights))
    p = rtcore.PtParams(rtcore.Camera(*S.BOX_CAMERA), w, h, spp, 0, depth, 3, seed, 0.0, 0)
    nb = ctx.pt_scratch_bytes(p)
    scratch = torch.empty(nb, dtype=torch.uint8, device="cuda")
    ob, _ = orc.build_blas([(v, i, None)])
    o = orc.path_trace(ob, tm, m, lights, S.BOX_CAMERA, w, h, spp, depth, 3, seed, 0.0)
    for _ in range(2):
        accum = torch.zeros(w * h * 16, dtype=torch.uint8, device="cuda")
        ctx.path_trace(sc, p, accum, scratch, nb)
        ctx.sync()
        assert host(accum).view(np.float32).tobytes() == o.tobytes()


@pytest.mark.parametrize("ring,threads", [(16, 128), (32, 256)])
def test_coincident_walls_in_a_batch_match_oracle(ctx, orc, ring, threads):
    import rtcore
    import rtcore.scenes as S
    import torch
    from rtcore.batch import GpuScene, SceneSpec, batch_params
    seed, spp, depth = 0x5EED0004, 4, 8
    specs = [SceneSpec("box", 480, 200, 150, S.BOX_CAMERA, 21), SceneSpec("box", 480, 160, 120, S.BOX_CAMERA, 22)]
    data = [_box_of_walls(sp.seed) for sp in specs]
    scenes = [GpuScene(ctx, sp, d) for sp, d in zip(specs, data)]
    table = [sc.batch_scene() for sc in scenes]
    p = batch_params(spp, depth, seed)
    t = rtcore.default_batch_tuning()
    t.stack_ring, t.trace_threads, t.trace_blocks_per_sm = ring, threads, 1024 // threads
    nb = ctx.batch_scratch_bytes(table, p, t)
    scratch = torch.empty(nb, dtype=torch.uint8, device="cuda")
    plan = ctx.batch_plan(table, p, scratch, nb, t)
    for sc in scenes:
        sc.accum.zero_()
    plan.launch(0)
    ctx.sync()
    plan.close()
    for sp, sc, (v, i, tm, m) in zip(specs, scenes, data):
        ob, _ = orc.build_blas([(v, i, None)])
        o = orc.path_trace(ob, tm, m, S.emissive_lights(v, i, tm, m), sp.camera, sp.width, sp.height, spp, depth, 3,
                           seed, p.ray_eps)
        assert host(sc.accum).view(np.float32).tobytes() == o.tobytes()
