"""Biases at the ends of FP32's range in cache inference, whose kernel adds a
bias as three BF16 parts: infinities, values that BF16 rounds to infinity, the
largest finite ones and the smallest, at the outputs and in a hidden layer."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import dev, host
from test_gpu_cache import FWD_TOL, cache, get_params, random_inputs  # noqa: F401

pytestmark = pytest.mark.gpu

MAX = np.finfo(np.float32).max
ROUNDS_UP = np.array([0x7F7F8000], np.uint32).view(np.float32)[0]  # halfway from BF16's largest to 2^128


def _query(ctx, cache, params, x):  # noqa: F811
    import torch
    ctx.cache_set_params(cache, torch.from_numpy(params).cuda())
    out = torch.empty(len(x) * 16, dtype=torch.uint8, device="cuda")
    ctx.cache_query(cache, dev(x), out, len(x))
    ctx.sync()
    return host(out).view(np.float32).reshape(-1, 4)[:, :3]


@pytest.mark.parametrize("bias", [np.inf, -np.inf, MAX, -MAX, ROUNDS_UP, -ROUNDS_UP, np.nextafter(ROUNDS_UP, np.float32(0))])
def test_output_bias_at_the_ends_of_the_range(ctx, cache, bias):  # noqa: F811
    from oracle import mlp
    x = random_inputs(300, 3)
    params = get_params(ctx, cache)
    plain = _query(ctx, cache, params, x)
    params[mlp.W_OFF[5][1] + 1] = bias
    y = _query(ctx, cache, params, x)
    # the other terms are far below the bias's last place
    assert (y[:, 1] == np.float32(bias)).all(), y[:3]
    assert y[:, [0, 2]].tobytes() == plain[:, [0, 2]].tobytes()


def test_hidden_unit_switched_off_by_its_bias(ctx, cache):  # noqa: F811
    from oracle import mlp
    x = random_inputs(300, 4)
    params = get_params(ctx, cache)
    params[mlp.W_OFF[2][1] + 5] = -np.inf  # ReLU leaves 0
    y = _query(ctx, cache, params, x)
    yo = mlp.forward(params, x, (-1, -1, -1), (1, 1, 1))[:, :3]
    assert np.isfinite(y).all()
    assert np.abs(y - yo).max() < FWD_TOL * np.abs(yo).max()


@pytest.mark.parametrize("exponent", [-149, -140, -127, -125, -110, -66, -62, -60, -58, -20, 0, 100])
def test_bias_alone_is_the_output(ctx, cache, exponent):  # noqa: F811
    """Output weights of 0: the outputs are the biases, to the last bit."""
    from oracle import mlp
    x = random_inputs(130, 5)
    params = get_params(ctx, cache)
    wo, bo = mlp.W_OFF[5]
    params[wo:bo] = 0
    rng = np.random.default_rng(exponent + 200)
    for _ in range(8):
        b = (rng.uniform(1, 2, 3) * 2.0 ** exponent * rng.choice([-1, 1], 3)).astype(np.float32)
        params[bo:bo + 3] = b
        y = _query(ctx, cache, params, x)
        assert (y == b).all(), (b, y[0])
