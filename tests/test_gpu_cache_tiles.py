"""The cache kernels at the edges of their tiles: training gradients where the
tile height changes (32, 64 and 128 rows) and with ragged last tiles, inference
with one row to several tiles per group and SM.  Bounds: those of
test_gpu_cache.py (BF16 roundings that flip where FP32 sums differ in their last
bits)."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import dev, host
from test_gpu_cache import FWD_TOL, GRAD_TOL, cache, get_params, random_inputs, smooth_target  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 2048, 2049, 9728, 9729])
def test_gradient_tiles_match_oracle(ctx, cache, n):  # noqa: F811
    from oracle import mlp
    import torch
    x = random_inputs(n, 40 + n)
    t = smooth_target(x)
    g = torch.empty(mlp.N_PARAMS * 4, dtype=torch.uint8, device="cuda")
    ctx.cache_gradient(cache, dev(x), dev(t), n, g)
    ctx.sync()
    gg = host(g).view(np.float32).astype(np.float64)
    go, _ = mlp.gradient(get_params(ctx, cache), x, t, (-1, -1, -1), (1, 1, 1))
    for L in range(6):
        wo, bo = mlp.W_OFF[L]
        for a, b in ((gg[wo:bo], go[wo:bo]), (gg[bo:bo + mlp.OUT[L]], go[bo:bo + mlp.OUT[L]])):
            assert np.abs(a - b).max() <= GRAD_TOL * max(np.abs(b).max(), 1e-30), L


@pytest.mark.parametrize("n", [1, 127, 129, 19456, 19457, 97281])
def test_query_tiles_match_oracle(ctx, cache, n):  # noqa: F811
    from oracle import mlp
    import torch
    x = random_inputs(n, 60 + n)
    out = torch.full(((n + 1) * 4,), -7.0, dtype=torch.float32, device="cuda")
    ctx.cache_query(cache, dev(x), out, n)
    ctx.sync()
    y = out.cpu().numpy().reshape(-1, 4)
    assert (y[n] == -7.0).all() and not (y[:n, 0] == -7.0).any()
    idx = np.unique(np.r_[0, np.linspace(0, n - 1, min(n, 1500)).astype(int), max(0, n - 130):n])
    yo = mlp.forward(get_params(ctx, cache), x[idx], (-1, -1, -1), (1, 1, 1))[:, :3]
    assert np.abs(y[idx, :3] - yo).max() < FWD_TOL * np.abs(yo).max()
