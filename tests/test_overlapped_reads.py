"""Kernels that a build or sort launches while the kernel before still runs
(programmatic dependent launch) read what that kernel writes through L2, never
through the read-only path: ld.global.nc promises nothing for memory that is
written while the grid is resident, even after griddepcontrol.wait.  Checked in
the sources, as no run shows it reliably."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "build-up-phase_gb300" / "csrc"

# Overlapped kernels and the device functions they read with, and their const
# __restrict__ parameters that no kernel of the chain writes (a caller's inputs).
FUNCTIONS = [("rt_sort.cu", "k_onesweep", ()), ("rt_build.cu", "k_morton", ()), ("rt_build.cu", "k_tree", ()),
             ("rt_build.cu", "k_tree_climb", ()), ("rt_build.cu", "climb_global", ()),
             ("rt_build.cu", "complete_node", ()), ("rt_build.cu", "tree_arrive", ()),
             ("rt_build.cu", "k_prep_inst", ("inst",))]


def _function(text, name):
    """(parameters, body) of the function's definition."""
    for m in re.finditer(rf"\b{name}\s*\(", text):
        depth, k = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[k], 0)
            k += 1
        params = text[m.end():k - 1]
        rest = text[k:].lstrip()
        if not rest.startswith("{"):
            continue  # a call
        start = text.index("{", k)
        depth, e = 1, start + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[e], 0)
            e += 1
        return params, text[start:e]
    raise AssertionError(f"no definition of {name}")


@pytest.mark.parametrize("file,name,inputs", FUNCTIONS)
def test_no_read_only_loads_of_what_the_kernel_before_writes(file, name, inputs):
    text = re.sub(r"//[^\n]*", "", (CSRC / file).read_text())
    params, body = _function(text, name)
    assert "__ldg(" not in body and "ldg4(" not in body
    for p in re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params):
        if p not in inputs:
            assert not re.search(rf"\b{p}\s*\[", body), f"{name} reads {p} as const __restrict__"


def test_every_overlapped_kernel_of_the_build_is_checked():
    names = {n for _, n, _ in FUNCTIONS}
    for file in ("rt_sort.cu", "rt_build.cu"):
        text = (CSRC / file).read_text()
        launched = set(re.findall(r"launch_pdl\((?:blas \? )?(k_\w+)", text))
        assert launched and launched - names <= {"k_prep_tris"}  # reads the caller's geometry alone
