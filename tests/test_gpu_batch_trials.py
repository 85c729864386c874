"""The batch autotuner times each kernel and launch shape once: stack rings of 8
and 16 are one kernel, so no two of its trials may differ in that alone."""
from __future__ import annotations

import json

import pytest

pytestmark = pytest.mark.gpu


def test_no_kernel_is_timed_under_two_names(ctx, tmp_path):
    import torch
    from rtcore.batch import GpuScene, SceneSpec, batch_params, host_scene
    specs = [SceneSpec("soup", 3000, 96, 64, ((0.5, 0.5, 2.2), 45.0), 1), SceneSpec("box", 2000, 64, 64, ((0, 0, 0.95), 60.0), 2)]
    scenes = [GpuScene(ctx, sp, host_scene(sp)) for sp in specs]
    table = [sc.batch_scene() for sc in scenes]
    p = batch_params(1, 4, 5)
    nb = ctx.batch_scratch_bytes(table, p)
    scratch = torch.empty(nb, dtype=torch.uint8, device="cuda")
    cache = tmp_path / "tune.json"
    ctx.batch_autotune(table, p, scratch, nb, cache)
    ctx.sync()
    trials = [t[0].replace("ring 8,", "ring 16,") for e in json.loads(cache.read_text())["entries"].values()
              for t in e["trials"]]
    assert len(trials) > 5
    assert len(set(trials)) == len(trials), trials
