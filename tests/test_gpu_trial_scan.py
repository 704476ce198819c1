"""Many external trials judged in one call are taken by a grid of blocks: each result must be, bit for
bit, that of the trial judged alone, for counts below, at and above the number of resident blocks."""
import numpy as np
import pytest

from ph_brush_b200 import Engine, configs

from test_gpu_energy import random_trials


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [128, 256])
@pytest.mark.parametrize("n", [1, 2, 295, 296, 297, 593, 1201])
def test_scan_equals_single_trials(n, threads):
    s, p = configs.small_system(seed=8)
    s.capacity += 8
    trials = random_trials(s, p, np.random.default_rng(5), n)
    with Engine(s, p) as e:
        e.set_tuning(16, threads)
        before = e.energy()[0]
        got = e.delta_energy_components(trials)
        dE = e.delta_energy(trials)
        for k in sorted({0, 1 % n, n // 2, n - 1}):
            assert got[k] == e.delta_energy_components([trials[k]])[0], k
            assert dE[k] == got[k]["total"]
        assert e.energy()[0] == before  # the state is left alone
