"""A negative number of external trials is refused by every call that takes one (its copies would be
sized by it), before anything is allocated or copied; none at all is no error; the engine goes on."""
import numpy as np
import pytest

from ph_brush_b200 import Engine, _abi, configs


@pytest.mark.gpu
def test_negative_trial_counts_are_refused():
    s, p = configs.small_system(seed=4)
    lib = _abi.lib()
    with Engine(s, p) as e:
        i = int(np.flatnonzero(s.flags & _abi.F_MOBILE)[0])
        move = [dict(index=i, x=float(s.x[i]), y=float(s.y[i]), z=float(s.z[i]), q=float(s.q[i]), type=int(s.type[i]))]
        t = (_abi.Trial * 1)(Engine.make_trial(move))
        dE = np.zeros(1)
        comp = (_abi.EnergyComponents * 1)()
        rows = np.zeros(4096, np.float32)
        for n, code in ((0, 0), (-1, 1), (-7, 1), (-2 ** 31, 1)):
            assert lib.phmc_delta_energy(e._h, 0, t, n, _abi.dptr(dE)) == code
            assert lib.phmc_delta_energy_components(e._h, 0, t, n, comp) == code
            assert lib.phmc_surrogate_describe(e._h, 0, t, n, _abi.fptr(rows), _abi.dptr(dE)) == code
        assert abs(e.delta_energy([move])[0]) <= 1e-4  # a move to where it is
