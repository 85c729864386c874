"""The radix tree built in blocks of 256 keys (k_tree) and across them
(k_tree_climb): sizes around the block, equal keys (ordered by index, subtrees
that span blocks), keys on a line (every node at a block's edge shares a long
prefix), and instances.  Byte-identical structures with the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import GpuBlas, GpuTlas, compare_accels, ptr_of, single_instance

pytestmark = pytest.mark.gpu


def _triangles(kind, n):
    import rtcore.scenes as S
    if kind == "soup":
        return S.soup(n, n)
    tri = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32) * np.float32(0.01)
    v = np.tile(tri, (n, 1))
    if kind == "line":
        v += np.repeat(np.linspace(0, 1, n, dtype=np.float32), 3)[:, None]
    return v, np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("kind", ["soup", "equal", "line"])
@pytest.mark.parametrize("n", [2, 255, 256, 257, 512, 513, 1025, 5000])
def test_tree_blocks_match_oracle(ctx, orc, kind, n):
    v, i = _triangles(kind, n)
    g = GpuBlas(ctx, [(v, i, None)])
    o, rc = orc.build_blas([(v, i, None)])
    assert rc == 0
    compare_accels(g.bytes(), o, 48)


@pytest.mark.parametrize("n", [256, 300])
def test_instance_tree_blocks_match_oracle(ctx, orc, n):
    v, i = _triangles("soup", 50)
    gb, (ob, _) = GpuBlas(ctx, [(v, i, None)]), orc.build_blas([(v, i, None)])

    def instances(ref):
        inst = np.concatenate([single_instance(ref) for _ in range(n)])
        inst["transform"][:, :, 3] = np.random.default_rng(n).uniform(-5, 5, (n, 3))
        return inst

    compare_accels(GpuTlas(ctx, instances(gb.addr)).bytes(), orc.build_tlas(instances(ptr_of(ob)))[0], 80,
                   ignore_ref=True)


@pytest.mark.parametrize("kind", ["soup", "equal", "line"])
@pytest.mark.parametrize("n", [25_600, 25_601])
def test_climb_in_one_block_or_many_matches_oracle(ctx, orc, kind, n):
    """100 blocks of keys: the largest tree whose rest one block climbs."""
    v, i = _triangles(kind, n)
    g = GpuBlas(ctx, [(v, i, None)])
    o, rc = orc.build_blas([(v, i, None)])
    assert rc == 0
    compare_accels(g.bytes(), o, 48)
