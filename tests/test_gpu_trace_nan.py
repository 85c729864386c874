"""Rays with NaN among their limits, origins and directions: no triangle is hit
within a NaN limit or an empty interval, and such a ray is a miss at once (an
all-NaN box test does not let it into every node); node visits and triangle
tests equal the oracle's, which compares as IEEE 754 does."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import GpuBlas, GpuTlas, dev, gpu_trace_any, gpu_trace_closest, gpu_trace_stats, ptr_of

pytestmark = pytest.mark.gpu


def _rays(seed, n):
    import rtcore.scenes as S
    rng = np.random.default_rng(seed)
    r = S.incoherent_rays(seed, n, (0, 0, 0), (1, 1, 1), 1e30)
    for name in ("org", "dir"):
        m = rng.random((n, 3)) < 0.25
        r[name][m] = rng.choice([np.nan, np.nan, np.inf, -np.inf, 0.0, -0.0], m.sum())
    m = rng.random(n) < 0.4
    r["tmin"][m] = rng.choice([np.nan, np.nan, np.inf, -np.inf, -1e30, 0.5], m.sum())
    m = rng.random(n) < 0.4
    r["tmax"][m] = rng.choice([np.nan, np.nan, np.inf, -np.inf, 0.0, 0.2], m.sum())
    return r


@pytest.mark.parametrize("instances", [0, 30])
def test_nan_rays_match_oracle(ctx, orc, instances):
    import rtcore.scenes as S
    from oracle import INSTANCE_DTYPE
    items = [(*S.soup(17, 5000), None)]
    g = GpuBlas(ctx, items)
    o, rc = orc.build_blas(items)
    assert rc == 0
    addr, oa = g.addr, o
    if instances:
        rng = np.random.default_rng(4)
        inst = np.zeros(instances, INSTANCE_DTYPE)
        for k in range(instances):
            inst[k]["transform"][:, :3] = np.linalg.qr(rng.normal(size=(3, 3)))[0]
            inst[k]["transform"][:, 3] = rng.uniform(-1, 1, 3)
        inst["custom_index_and_mask"] = 0xFF << 24
        inst["accel_ref"] = g.addr
        gt = GpuTlas(ctx, inst)
        inst["accel_ref"] = ptr_of(o)
        oa, rc = orc.build_tlas(inst)
        assert rc == 0
        addr = gt.addr
    rays = _rays(3, 20_000)
    hg, xg = gpu_trace_closest(ctx, addr, rays, ext=True)
    ho, so, xo = orc.trace_closest(oa, rays, ext=True)
    assert hg.tobytes() == ho.tobytes()
    assert xg.tobytes() == xo.tobytes()
    occ, sa = orc.trace_any(oa, rays)
    np.testing.assert_array_equal(gpu_trace_any(ctx, addr, rays), occ)
    np.testing.assert_array_equal(gpu_trace_stats(ctx, addr, rays), so)
    np.testing.assert_array_equal(gpu_trace_stats(ctx, addr, rays, any_hit=True), sa)


def test_nan_limits_walk_nothing(ctx):
    """Rays of NaN alone take no longer than others (they walked the whole tree)."""
    import rtcore.scenes as S
    import torch
    g = GpuBlas(ctx, [(*S.soup(18, 200_000), None)])
    n = 20_000
    rays = np.zeros(n, S.RAY_DTYPE)
    for name in ("org", "dir", "tmin", "tmax"):
        rays[name] = np.nan
    good = S.incoherent_rays(5, n, (0, 0, 0), (1, 1, 1), 1e30)
    hits = torch.empty(n * 16, dtype=torch.uint8, device="cuda")

    def ms(r):
        d = dev(r)
        t = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            ctx.trace_closest(g.addr, d, hits, n)
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b))
        return float(np.median(t))

    assert ms(rays) < ms(good)
    ctx.sync()
