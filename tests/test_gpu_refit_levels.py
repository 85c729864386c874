"""Refit by levels (rt_refit_blas): trees whose levels are all small (one block),
mixed, and deep with internal nodes of every level listed out of order; leaves
of several records; unlike sizes around a warp's 32 nodes.  Byte-identical with
the oracle's refit."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import GpuBlas, compare_accels

pytestmark = pytest.mark.gpu


def _moved(v, seed):
    rng = np.random.default_rng(seed)
    return (v + rng.uniform(-0.02, 0.02, v.shape)).astype(np.float32)


@pytest.mark.parametrize("scene", ["soup 33", "soup 130", "soup 5001", "box 1 4", "box 3 20", "copies 400"])
def test_refit_levels_match_oracle(ctx, orc, scene):
    import rtcore.scenes as S
    kind, *a = scene.split()
    if kind == "soup":
        v, i = S.soup(31, int(a[0]))
    elif kind == "box":
        v, i = S.box(9, int(a[0]), int(a[1]))[:2]
    else:  # equal keys: a deep, narrow tree
        v = np.tile(np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32), (int(a[0]), 1))
        i = np.arange(len(v), dtype=np.uint32).reshape(-1, 3)
    g = GpuBlas(ctx, [(v, i, None)])
    o, rc = orc.build_blas([(v, i, None)])
    assert rc == 0
    for seed in (1, 2):  # twice: nothing of the first refit may stay behind
        moved = [(_moved(v, seed), i, None)]
        g.refit(ctx, moved)
        assert orc.refit_blas(o, moved) == 0
        compare_accels(g.bytes(), o, 48)
