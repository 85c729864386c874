"""Instances without a structure (accel_ref 0, which a build takes as empty):
nothing enters them, rays of NaNs included, whose box tests let them into
everything.  The same hits, frame and counts as with an empty structure there."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import GpuBlas, GpuTlas, gpu_trace_any, gpu_trace_closest, gpu_trace_stats, host

pytestmark = pytest.mark.gpu


def _tlas(ctx, blas, nothing):
    from oracle import INSTANCE_DTYPE
    rng = np.random.default_rng(6)
    inst = np.zeros(30, INSTANCE_DTYPE)
    inst["transform"] = np.eye(4, dtype=np.float32)[:3]
    inst["transform"][:, :, 3] = rng.uniform(-1, 1, (30, 3))
    inst["custom_index_and_mask"] = np.arange(30) | (0xFF << 24)
    inst["accel_ref"] = np.where(np.arange(30) % 3 == 1, nothing, blas.addr)
    return GpuTlas(ctx, inst)


def test_instances_without_a_structure(ctx):
    import rtcore
    import rtcore.scenes as S
    import torch
    blas = GpuBlas(ctx, [(*S.soup(3, 400), None)])
    empty = GpuBlas(ctx, [(np.zeros((0, 3), np.float32), np.zeros((0, 3), np.uint32), None)])
    rays = S.incoherent_rays(9, 6000, (-1, -1, -1), (2, 2, 2), 1e30)
    rays["org"][::4] = np.nan  # finite limits: every box test passes
    rays["dir"][1::8] = np.nan
    got = []
    for nothing in (0, empty.addr):
        t = _tlas(ctx, blas, nothing)
        h, x = gpu_trace_closest(ctx, t.addr, rays, ext=True)
        image = torch.zeros(64 * 48 * 4, dtype=torch.float32, device="cuda")
        p = rtcore.sample_pipeline(rtcore.RT_CHIT_BARYCENTRIC)
        ctx.trace_rays(p, None, t.addr, rtcore.Camera((float("nan"), 0.0, 4.0), 60.0), image, 64, 48)
        ctx.sync()
        got.append([h.tobytes(), x.tobytes(), gpu_trace_any(ctx, t.addr, rays).tobytes(),
                    gpu_trace_stats(ctx, t.addr, rays).tobytes(), host(image).tobytes()])
    assert got[0] == got[1]
