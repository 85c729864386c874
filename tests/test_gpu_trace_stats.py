"""rt_trace_stats: node visits and triangle tests equal the oracle's for one- and
two-level structures, closest and any hit, at ray counts around a lane, a warp
and the grid; and the counting walk costs about what the query does."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import GpuBlas, GpuTlas, dev, gpu_trace_stats, ptr_of

pytestmark = pytest.mark.gpu


def _scene(ctx, orc, kind):
    import rtcore.scenes as S
    from oracle import INSTANCE_DTYPE
    items = [[(*S.soup(5, 4000), None)], [(*S.box(6, 2, 6)[:2], None)],
             [(np.zeros((0, 3), np.float32), np.zeros((0, 3), np.uint32), None)]]
    gb = [GpuBlas(ctx, it) for it in items]
    ob = [orc.build_blas(it)[0] for it in items]
    if kind != "instances":
        k = {"soup": 0, "empty": 2}[kind]
        return gb[k].addr, ob[k], (gb, ob)
    rng = np.random.default_rng(3)
    inst = np.zeros(40, INSTANCE_DTYPE)
    for k in range(40):
        q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        inst[k]["transform"][:, :3] = q * rng.uniform(0.3, 0.8)
        inst[k]["transform"][:, 3] = rng.uniform(0, 2, 3)
    which = np.arange(40) % 3
    inst["custom_index_and_mask"] = np.where(np.arange(40) % 7 == 3, 0, 0xFF << 24)
    inst["accel_ref"] = [gb[w].addr for w in which]
    gt = GpuTlas(ctx, inst)
    inst["accel_ref"] = [ptr_of(ob[w]) for w in which]
    ot, rc = orc.build_tlas(inst)
    assert rc == 0
    return gt.addr, ot, (gb, ob, gt)


@pytest.mark.parametrize("kind", ["soup", "instances", "empty"])
@pytest.mark.parametrize("n", [1, 33, 4097, 150_001])
def test_counts_match_oracle(ctx, orc, kind, n):
    import rtcore.scenes as S
    addr, o, keep = _scene(ctx, orc, kind)
    rays = S.incoherent_rays(n, n, (0, 0, 0), (2, 2, 2), 1e30)
    rays["tmax"][::3] = 0.3
    np.testing.assert_array_equal(gpu_trace_stats(ctx, addr, rays), orc.trace_closest(o, rays)[1])
    np.testing.assert_array_equal(gpu_trace_stats(ctx, addr, rays, any_hit=True), orc.trace_any(o, rays)[1])


def test_counting_costs_about_a_query(ctx):
    """Same rays, same structure; a walk with one thread per ray took 2.7 times
    the query's time."""
    import rtcore.scenes as S
    import torch
    g = GpuBlas(ctx, [(*S.soup(8, 300_000), None)])
    n = 2_000_000
    rays = dev(S.incoherent_rays(8, n, (0, 0, 0), (1, 1, 1), 1e30))
    hits = torch.empty(n * 16, dtype=torch.uint8, device="cuda")
    c = torch.zeros(2, dtype=torch.int64, device="cuda")

    def us(call):
        t = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            call()
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b))
        return float(np.median(t))

    query = us(lambda: ctx.trace_closest(g.addr, rays, hits, n))
    stats = us(lambda: ctx.trace_stats(g.addr, rays, n, False, c))
    print(f"query {query:.3f} ms, statistics {stats:.3f} ms")
    assert stats < 2.0 * query
