"""Coincident axis-parallel triangles: their boxes have no thickness, so which
of two equally near ones the far limit still admits depends on the order of the
tests; the persistent traversal, which tests records in batches, has to give the
oracle's answer, and the same one each time."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import GpuBlas, gpu_trace_closest

pytestmark = pytest.mark.gpu


def _walls(seed, walls=60, copies=12):
    """Axis-parallel triangles, each with copies on it, beside it in its plane
    and a rounding error off it."""
    rng = np.random.default_rng(seed)
    tris = []
    for _ in range(walls):
        axis = rng.integers(3)
        centre, t = rng.uniform(-1, 1, 3), rng.uniform(-2, 2, (3, 3))
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


@pytest.mark.parametrize("seed", [2, 5])
def test_coincident_walls_match_oracle(ctx, orc, seed):
    import rtcore.scenes as S
    items = [_walls(seed)]
    g = GpuBlas(ctx, items)
    ob, rc = orc.build_blas(items)
    assert rc == 0
    n = 1_000_000
    rays = S.incoherent_rays(seed, n, (-1, -1, -1), (1, 1, 1), 1e30)
    rays["org"][::7, 0] = 0.0  # limits of -0 at the ray's own origin
    rays["tmin"][::7] = -0.0
    rays["tmax"][::7] = -0.0
    ho, _, xo = orc.trace_closest(ob, rays, ext=True)
    for _ in range(2):
        hg, xg = gpu_trace_closest(ctx, g.addr, rays, ext=True)
        assert hg.tobytes() == ho.tobytes()
        assert xg.tobytes() == xo.tobytes()
