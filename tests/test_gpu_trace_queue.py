"""The persistent traversal's triangle queue (records tested in batches by the
whole warp) and its spreading of few rays over many warps, against the oracle:
ray counts around a lane, a warp and the whole grid; leaves of several
triangles; coincident triangles, whose hits tie."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import GpuBlas, gpu_trace_any, gpu_trace_closest

pytestmark = pytest.mark.gpu


def _coincident(n=48):
    """n copies of one triangle and n of another behind it: every hit ties."""
    a = np.array([[-1, -1, 0], [1, -1, 0], [0, 1, 0]], np.float32)
    v = np.concatenate([np.tile(a, (n, 1)), np.tile(a + np.float32([0, 0, -0.5]), (n, 1))])
    order = np.random.default_rng(3).permutation(2 * n).astype(np.uint32)
    return v, (3 * order[:, None] + np.arange(3, dtype=np.uint32)).astype(np.uint32)


def _scene(name):
    import rtcore.scenes as S
    if name == "soup":
        return (*S.soup(21, 700), (0, 0, 0), (1, 1, 1))
    if name == "box":  # smooth meshes: leaves of up to three triangles
        return (*S.box(5, 3, 8)[:2], (-1, -1, -1), (1, 1, 1))
    return (*_coincident(), (-1, -1, -1), (1, 1, 1))


@pytest.mark.parametrize("name", ["soup", "box", "coincident"])
@pytest.mark.parametrize("n", [1, 31, 33, 4097, 175_105])
def test_batched_triangle_tests_match_oracle(ctx, orc, name, n):
    import rtcore.scenes as S
    v, i, lo, hi = _scene(name)
    g = GpuBlas(ctx, [(v, i, None)])
    ob, rc = orc.build_blas([(v, i, None)])
    assert rc == 0
    rays = S.incoherent_rays(100 + n, n, lo, hi, 1e30)
    rays["tmax"][::3] = 0.4  # limits inside the scene
    hg, xg = gpu_trace_closest(ctx, g.addr, rays, ext=True)
    ho, _, xo = orc.trace_closest(ob, rays, ext=True)
    assert hg.tobytes() == ho.tobytes()
    assert xg.tobytes() == xo.tobytes()
    np.testing.assert_array_equal(gpu_trace_any(ctx, g.addr, rays), orc.trace_any(ob, rays)[0])
