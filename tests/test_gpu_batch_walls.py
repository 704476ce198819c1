"""Batched trials in a thin slab: an accepted displacement moves a particle that a later trial of the
same batch displaces again, and whether the walls refuse that trial depends on the place it starts
from.  A few mobile ions between walls a little more than one step apart meet this in most batches;
every trial is followed by the oracle's one-at-a-time Monte Carlo (dE, infinite against finite, the
decisions replayed, final positions), alone (batches of 16) and beside 149 others (batches of 8)."""
import numpy as np
import pytest

from oracle import pyoracle as O
from ph_brush_b200 import Engine, _abi, configs
from ph_brush_b200.model import SystemArrays

from test_gpu_mc import de_close

HEIGHT, STEP, TRIALS = 2.5, 1.6, 800


def thin_slab(n, seed):
    """n / 2 ions of either charge between walls, in a box wide enough that few lie within a cutoff."""
    rng = np.random.default_rng(seed)
    L, cols = 40.0, int(np.ceil(np.sqrt(n)))
    k = np.arange(n)
    s = SystemArrays(((k % cols + 0.5) * L / cols).astype(np.float32), ((k // cols + 0.5) * L / cols).astype(np.float32),
                     rng.uniform(0.2, HEIGHT - 0.2, n).astype(np.float32), np.where(k % 2, -1.0, 1.0).astype(np.float32),
                     np.where(k % 2, 2, 3).astype(np.int32),
                     np.where(k % 2, _abi.F_MOBILE | _abi.F_ANION, _abi.F_MOBILE | _abi.F_CATION).astype(np.int32),
                     np.zeros(0, np.int32), np.zeros(0, np.int32), np.array([L, L, 24.0]), capacity=n + 4)
    p = configs.native_params(7.0, 7.0, (32, 32, 24), HEIGHT, seed, rc=2.0, p_disp=1.0, p_titr=0.0, disp_max=STEP)
    p.pending_max = 48
    return s, p


def picked(seed, t, n):
    """The particle (in list order) that trial t displaces."""
    w = O.philox((seed & 0xffffffff, seed >> 32), (t & 0xffffffff, t >> 32, 0, 0))
    return (int(w[1]) * n) >> 32


@pytest.mark.gpu
@pytest.mark.parametrize("replicas", [1, 150])
@pytest.mark.parametrize("n", [2, 12])
def test_wall_verdicts_follow_the_trials_before(n, replicas):
    s, p = thin_slab(n, seed=31 + n)
    with Engine([s] * replicas, [p] * replicas) as e:
        e.set_quorum(1.0)
        mv, dE, acc = e.set_trial_log(TRIALS)
        e.run(TRIALS)
        got = e.state(0)
    mc = O.MC(s, p)
    moved, repeats = {}, 0  # trials of each particle's last accepted move
    for t in range(TRIALS):
        m, d, _ = mc.step(int(acc[t]))
        assert m == mv[t]
        if np.isfinite(d) and np.isfinite(dE[t]):
            assert de_close(dE[t], d), (t, d, dE[t])
        else:
            assert np.isinf(d) == np.isinf(dE[t]) or min(d, dE[t]) > 1e6, (t, d, dE[t])
        i = picked(p.seed, t, n)
        repeats += bool(np.isinf(d) and t - moved.get(i, -99) < 16)
        if acc[t]:
            moved[i] = t
    assert repeats > 20 and acc.sum() > 200
    ref = mc.state()
    for k in ("x", "y", "z"):
        assert np.array_equal(got[k][:n], ref[k][:n]), k
