"""The collapse's shortcuts (widening from whole tables, slot rounds that end
when the least slots differ) and its hand-over from block 0 to the grid: node
counts around 64 and 512 per level, every width, regular grids whose areas and
slot costs tie, flat geometry (zero areas).  Byte-identical with the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import GpuBlas, compare_accels

pytestmark = pytest.mark.gpu


def _lattice(side, flat):
    """One small triangle per lattice point: equal boxes, tied areas and costs."""
    z = np.zeros(1) if flat else np.arange(side)
    p = np.stack(np.meshgrid(np.arange(side), np.arange(side), z, indexing="ij"), -1).reshape(-1, 3).astype(np.float32)
    tri = np.array([[0, 0, 0], [0.25, 0, 0], [0, 0.25, 0]], np.float32)
    v = (p[:, None, :] + tri[None]).reshape(-1, 3)
    return v, np.arange(len(v), dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("width", [4, 5, 8])
@pytest.mark.parametrize("scene", ["soup 600", "soup 5000", "soup 40000", "lattice 16", "flat 64"])
def test_collapse_paths_match_oracle(ctx, orc, scene, width):
    import rtcore
    import rtcore.scenes as S
    kind, n = scene.split()
    v, i = S.soup(77, int(n)) if kind == "soup" else _lattice(int(n), kind == "flat")
    flags = rtcore.build_width(width)
    g = GpuBlas(ctx, [(v, i, None)], flags)
    o, rc = orc.build_blas([(v, i, None)], flags)
    assert rc == 0
    compare_accels(g.bytes(), o, 48)
