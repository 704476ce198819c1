"""The network's gradient at the edges of its kernels' tiles: hidden sizes whose column pairs do not
divide a block, sample counts below one block's rows and just past a GEMM tile.  Against the
BF16-emulating oracle, at the repository's tolerance (1 % relative norm)."""
import numpy as np
import pytest

from oracle import surrogate_oracle as SO
from ph_brush_b200 import Surrogate

from test_surrogate import K, random_samples


@pytest.mark.gpu
@pytest.mark.parametrize("hidden", [16, 48, 112, 128])
@pytest.mark.parametrize("n", [1, 31, 33, 129, 520])
def test_gradient_at_tile_edges(hidden, n):
    rng = np.random.default_rng(100 * hidden + n)
    x, sign, t = random_samples(rng, n)
    s = Surrogate(hidden=hidden, seed=4)
    mu, sd = x.reshape(-1, K).mean(0), x.reshape(-1, K).std(0) + 1.0
    s.set_scaling(mu, sd, 3.0)
    loss, g = s.gradient(x, sign, t)
    ref_loss, ref = SO.loss_grad(s.params(), K, hidden, mu.astype(np.float32), sd.astype(np.float32), 3.0, x, sign, t, 25.0, bf=True)
    assert abs(loss - ref_loss) <= 1e-2 * abs(ref_loss)
    assert np.linalg.norm(g - ref) <= 1e-2 * np.linalg.norm(ref)
    again = s.gradient(x, sign, t)[1]  # the tickets are back at zero, the sums in a fixed order
    assert np.array_equal(g, again)
