"""A cell that overflows while a batch's accepted moves are entered stops the replica there: no
trial beyond that batch is judged, whatever the timing, so the state left behind is the one after it.
Ideal particles, one per cell at most, so every move is accepted and batches end only at a particle
drawn twice; positions against the oracle's Monte Carlo (the same proposal stream)."""
import numpy as np
import pytest

from oracle import pyoracle as O
from ph_brush_b200 import Engine, _abi, configs
from ph_brush_b200.model import SystemArrays

from test_gpu_batch_walls import picked

N, L = 2000, 40


def ideal_gas(seed):
    """N neutral particles in the centres of N of the 40^3 unit cells, no walls."""
    rng = np.random.default_rng(seed)
    c = rng.choice(L ** 3, N, replace=False)
    z = np.zeros(N, np.float32)
    s = SystemArrays((c % L + 0.5).astype(np.float32), (c // L % L + 0.5).astype(np.float32),
                     (c // (L * L) + 0.5).astype(np.float32), z, np.zeros(N, np.int32), np.full(N, _abi.F_MOBILE, np.int32),
                     np.zeros(0, np.int32), np.zeros(0, np.int32), np.array([L, L, L], float), capacity=N + 4)
    p = configs.native_params(7.0, 7.0, (16, 16, 16), 0.0, seed, p_disp=1.0, p_titr=0.0, disp_max=0.9, lb=0.0)
    p.lj_eps = p.lj_eps * 0.0
    p.cell_cap = 1
    return s, p


@pytest.mark.gpu
@pytest.mark.parametrize("seed", [1, 2, 3])
@pytest.mark.parametrize("replicas,batch", [(1, 16), (150, 8)])
def test_no_trial_beyond_the_batch_of_an_overflow(replicas, batch, seed):
    s, p = ideal_gas(seed)
    with Engine([s] * replicas, [p] * replicas) as e:
        e.set_quorum(1.0)
        with pytest.raises(_abi.PhmcError) as ei:
            e.run(4000)
        assert ei.value.code == 3
        got = e.state(0)
    mc = O.MC(s, p)
    cell = lambda st: tuple(np.minimum((st[k][:N]).astype(int), L - 1) for k in ("x", "y", "z"))
    occ = np.zeros((L, L, L), int)
    np.add.at(occ, cell(mc.state()), 1)
    full, beyond, t = False, 0, 0  # trials after the one that overflows a cell; all
    while True:
        st = mc.state()
        if full and all(np.array_equal(got[k][:N], st[k][:N]) for k in ("x", "y", "z")):
            break  # the state that the engine left behind
        assert beyond < batch, "trials were judged beyond the overflow's batch"
        beyond += full
        i, was = picked(p.seed, t, N), cell(st)
        assert mc.step()[2] == 1
        t += 1
        was, now = tuple(a[i] for a in was), tuple(a[i] for a in cell(mc.state()))
        if was != now and not full:
            occ[was] -= 1
            full = occ[now] >= p.cell_cap
            occ[now] += 1
