"""The bias gradients are sums over thousands of rows: no further from 64 bits than FP32 sums in 256
strided parts (rows k, k + 256, ... one after the other, the parts as a tree).  A network whose weights
are zero but for the last layer's makes the summed values known: dZ3 = bf16(dy w4 gelu'(0)), dy = -sign t / n,
signs drawn about one, so that the sums grow along the rows; root mean square over the columns."""
import numpy as np
import pytest
import torch

from ph_brush_b200 import Surrogate

from test_surrogate import K


def chain(a):
    s = np.zeros(a.shape[1:], np.float32)
    for row in a:
        s = s + row
    return s


def strided(x):
    n = len(x) // 256 * 256
    p = chain(x[:n].reshape(-1, 256, x.shape[1]))
    p[:len(x) - n] += x[n:]
    p = p.reshape(8, 32, -1)
    for o in (16, 8, 4, 2, 1):
        p = p + p[:, np.arange(32) ^ o]
    return chain(p[:, 0])


@pytest.mark.gpu
@pytest.mark.parametrize("hidden", [128, 48])
@pytest.mark.parametrize("n", [4096, 5000, 16384])
def test_bias_sums_are_as_accurate_as_strided_ones(hidden, n):
    rng = np.random.default_rng(n + hidden)
    H = hidden
    s = Surrogate(hidden=H, seed=1)
    w4 = torch.linspace(1.0, 2.0, H).bfloat16().float().numpy()
    p = np.zeros(s.n_params, np.float32)
    off_b3, off_w4 = K * H + H + H * H + H + H * H, K * H + H + H * H + H + H * H + H
    p[off_w4:off_w4 + H] = w4
    s.set_params(p)
    s.set_scaling(np.zeros(K), np.ones(K), 1.0)
    t = rng.uniform(0.5, 1.0, n).astype(np.float32)
    sign = rng.normal(1.0, 1.0, (n, 4)).astype(np.float32)
    _, g = s.gradient(np.zeros((n, 4, K), np.float32), sign, t)
    dy = (sign * -t[:, None] / np.float32(n)).reshape(-1)
    dz = torch.from_numpy(dy[:, None] * w4[None] * np.float32(0.5)).bfloat16().float().numpy()
    exact = dz.astype(np.float64).sum(0)
    rms = lambda v: np.sqrt(np.mean((v - exact) ** 2))
    got = g[off_b3:off_b3 + H]
    assert np.allclose(got, exact, rtol=1e-5)
    assert rms(got) <= rms(strided(dz)), (rms(got), rms(strided(dz)))
    assert abs(g[-1] - dy.astype(np.float64).sum()) <= 1e-6 * abs(dy).sum()
