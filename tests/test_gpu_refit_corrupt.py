"""Refit of a structure whose nodes were damaged after the build (a file cut or
overwritten, memory written by something else): every reference a node holds is
checked before it is followed, and RT_ERR_BOUNDS is reported."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import NODE_DTYPE, GpuBlas, dev, header

pytestmark = pytest.mark.gpu


def _levels(nodes):
    """First node of each level of the breadth-first order, and the end."""
    lo, hi, out = 0, 1, [0]
    while hi < len(nodes):
        k = lo + np.nonzero(nodes["imask"][lo:hi])[0][-1]
        lo, hi = hi, int(nodes["child_base"][k]) + int(nodes["imask"][k]).bit_count()
        out.append(lo)
    return out + [hi]


def _damaged(nodes, damage):
    lv = _levels(nodes)
    if damage in ("child base", "child base past the end"):
        # an internal node that does not end its level: the levels stay as they are
        k = lv[1] + np.nonzero(nodes["imask"][lv[1]:lv[2]])[0][0]
        nodes["child_base"][k] = 0xFFFFFFFF if damage == "child base" else len(nodes)
    else:
        k = np.nonzero(nodes["imask"] == 0)[0][3]
        nodes["prim_base"][k] = {"record base": 0xFFFFFFFF, "record base, second": 0xFFFFFFFE}[damage]


@pytest.mark.parametrize("damage", ["child base", "child base past the end", "record base", "record base, second"])
def test_damaged_references_are_reported(ctx, damage):
    import rtcore
    import rtcore.scenes as S
    v, i = S.soup(12, 3000)
    g = GpuBlas(ctx, [(v, i, None)])
    buf = g.bytes().copy()
    h = header(buf)
    lo, hi = int(h["node_offset"]), int(h["node_offset"]) + 80 * int(h["node_count"])
    nodes = buf[lo:hi].view(NODE_DTYPE)
    assert len(nodes) > 100
    _damaged(nodes, damage)
    g.accel[:len(buf)].copy_(dev(buf))
    with pytest.raises(rtcore.RtError) as e:
        g.refit(ctx, [(v, i, None)])
    assert e.value.code == rtcore.RT_ERR_BOUNDS
    # the context goes on
    g2 = GpuBlas(ctx, [(v, i, None)])
    built = g2.bytes().copy()
    g2.refit(ctx, [(v, i, None)])
    assert g2.bytes().tobytes() == built.tobytes()


@pytest.mark.parametrize("n", [1, 3000])
def test_children_below_the_last_level_are_reported(ctx, n):
    import rtcore
    import rtcore.scenes as S
    v, i = S.soup(13, n)
    g = GpuBlas(ctx, [(v, i, None)])
    buf = g.bytes().copy()
    h = header(buf)
    lo, hi = int(h["node_offset"]), int(h["node_offset"]) + 80 * int(h["node_count"])
    nodes = buf[lo:hi].view(NODE_DTYPE)
    nodes["imask"][-1] |= 1  # the last node's first slot as an internal child
    g.accel[:len(buf)].copy_(dev(buf))
    with pytest.raises(rtcore.RtError) as e:
        g.refit(ctx, [(v, i, None)])
    assert e.value.code == rtcore.RT_ERR_BOUNDS
