"""The build's sort in tiles of 1,536 keys (small trees) and of 7,168: sizes
around both tiles and around the line between them, 30- and 63-bit keys (four
and eight passes), and builds that follow one another on the same scratch, whose
launches overlap.  Byte-identical structures with the oracle."""
from __future__ import annotations

import pytest

from helpers import GpuBlas, compare_accels

pytestmark = pytest.mark.gpu

MORTON30 = 1 << 8


@pytest.mark.parametrize("flags", [0, MORTON30])
@pytest.mark.parametrize("n", [1, 1535, 1536, 1537, 3073, 7168, 7169, 524_288, 524_289])
def test_sort_tiles_match_oracle(ctx, orc, n, flags):
    import rtcore.scenes as S
    items = [(*S.soup(n, n), None)]
    o, rc = orc.build_blas(items, flags)
    assert rc == 0
    g = GpuBlas(ctx, items, flags)
    geoms = g._geoms(items, g.keep)
    for _ in range(3):
        ctx.build_blas(geoms, flags, g.accel, g.sizes.accel_bytes, g.scratch, g.sizes.scratch_bytes, None)
    ctx.sync()
    compare_accels(g.bytes(), o, 48)
