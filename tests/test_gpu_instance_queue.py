"""The two-level traversal, whose lanes stop for instances and are served
together, against the oracle: ray counts around a lane, a warp and the grid;
coincident instances and triangles, whose hits tie; long runs of masked and
empty instances; hits at t = 0 under a far limit of -0."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import GpuBlas, GpuTlas, gpu_trace_any, gpu_trace_closest, ptr_of

pytestmark = pytest.mark.gpu

EMPTY = [(np.zeros((0, 3), np.float32), np.zeros((0, 3), np.uint32), None)]


def _layers(n):
    """n triangles in each of two parallel planes, the same triangle n times."""
    a = np.array([[-1, -1, 0], [1, -1, 0], [0, 1, 0]], np.float32)
    v = np.concatenate([np.tile(a, (n, 1)), np.tile(a - np.float32([0, 0, 0.5]), (n, 1))])
    order = np.random.default_rng(n).permutation(2 * n).astype(np.uint32)
    return v, (3 * order[:, None] + np.arange(3, dtype=np.uint32)).astype(np.uint32), None


def _instances(kind):
    """Object of each instance (0 layers, 1 soup, 2 empty) and its mask."""
    from oracle import INSTANCE_DTYPE
    n = {"coincident": 20, "skipped": 90, "spread": 40}[kind]
    rng = np.random.default_rng(n)
    inst = np.zeros(n, INSTANCE_DTYPE)
    inst["transform"] = np.eye(4, dtype=np.float32)[:3]
    which, mask = np.zeros(n, int), np.full(n, 0xFF)
    if kind == "skipped":  # one in 30 can be hit
        which = np.where(np.arange(n) % 2 == 0, 2, 0)
        mask = np.where(np.arange(n) % 2 == 1, 0, 0xFF)
        which[7::30], mask[7::30] = 0, 0xFF
    if kind == "spread":
        which = np.arange(n) % 2
        inst["transform"][:, :, 3] = rng.uniform(-1, 1, (n, 3))
    inst["custom_index_and_mask"] = np.arange(n) | (mask << 24)
    return inst, which


@pytest.mark.parametrize("kind", ["coincident", "skipped", "spread"])
@pytest.mark.parametrize("n", [1, 31, 33, 4097, 116_800])
def test_stopped_lanes_match_oracle(ctx, orc, kind, n):
    import rtcore.scenes as S
    items = [[_layers(24)], [(*S.soup(9, 300), None)], EMPTY]
    gb = [GpuBlas(ctx, it) for it in items]
    ob = [orc.build_blas(it)[0] for it in items]
    inst, which = _instances(kind)
    inst["accel_ref"] = [gb[w].addr for w in which]
    gt = GpuTlas(ctx, inst)
    inst["accel_ref"] = [ptr_of(ob[w]) for w in which]
    ot, rc = orc.build_tlas(inst)
    assert rc == 0
    rays = S.incoherent_rays(n, n, (-1, -1, -1), (1, 1, 1), 1e30)
    rays["tmax"][::3] = 0.4  # limits inside the scene
    flat = rays[1::5]        # from the plane of the first layer, far limit -0
    flat["org"][:, 2] = 0.0
    flat["tmin"] = -0.0
    flat["tmax"] = -0.0
    rays[1::5] = flat
    hg, xg = gpu_trace_closest(ctx, gt.addr, rays, ext=True)
    ho, _, xo = orc.trace_closest(ot, rays, ext=True)
    assert hg.tobytes() == ho.tobytes()
    assert xg.tobytes() == xo.tobytes()
    np.testing.assert_array_equal(gpu_trace_any(ctx, gt.addr, rays), orc.trace_any(ot, rays)[0])
    # the layers alone, one level
    hb = gpu_trace_closest(ctx, gb[0].addr, rays)
    assert hb.tobytes() == orc.trace_closest(ob[0], rays)[0].tobytes()
