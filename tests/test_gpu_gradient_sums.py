"""Length of the closure's weight- and bias-gradient sums on an 80^3 grid, where
each is exactly known: with the third layer's weights zero, the last layer's
input is constant per channel, so its bias gradient is the sum of the output
gradient and its weight gradients are that sum times the constants.

Biases are FP32 sums: the last, about 20 sequential additions of block partials,
round to sqrt(20 / 3) 2^-24 = 1.5e-7 of the terms' magnitude; bound 4 2^-24.
Weights are sums of the tensor core, whose additions drop on average half a
2^-23 of the partial sum, itself half of the whole on average: 4000 tiles of 8
steps over 148 blocks in two halves are 112 additions, 112 2^-25."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _bf16(x):
    return torch.from_numpy(np.asarray(x, np.float32)).to(torch.bfloat16).double().numpy()


@pytest.mark.parametrize("mean", [0.0, 0.5])
def test_sums_of_the_last_layer(mean):
    from lbman3d_b200.closure import Closure
    from oracle import closure as K
    grid = (80, 80, 80)
    V = grid[0] * grid[1] * grid[2]
    r = np.random.default_rng(V)
    with Closure(*grid, seed=1) as c:
        p = (0.02 * r.standard_normal(c.params().size)).astype(np.float32)
        (w2, b2), (w3, b3) = K.OFFSETS[2], K.OFFSETS[3]
        p[w2:b2] = 0
        p[b2:b2 + 32] = r.uniform(0.1, 1.5, 32)
        c.set_params(p)
        x, t = (r.standard_normal((n, V)).astype(np.float32) for n in (9, 8))
        x[0] += 1
        t += np.float32(mean)
        inv = (np.float32(1) / c.scales()[2]).astype(np.float64)[:, None]
        out = c.forward(x).astype(np.float64)
        _, g = c.gradient(x, t)
    d = (out - t * inv).astype(np.float32)  # the output gradient, as it is rounded
    go = _bf16(np.float32(2.0) / (np.float32(8.0) * np.float32(V)) * d)
    total, size = go.sum(axis=1), np.abs(go).sum(axis=1)
    assert np.max(np.abs(g[b3:b3 + 8] - total) / size) <= 4 * 2.0 ** -24
    act = torch.nn.functional.gelu(torch.from_numpy(p[b2:b2 + 32]).double()).float().to(torch.bfloat16).double().numpy()
    w = g[w3:b3].astype(np.float64).reshape(27, 32, 16)[:, :, :8]
    assert np.max(np.abs(w - act[:, None] * total) / (act[:, None] * size)) <= 112 * 2.0 ** -25
