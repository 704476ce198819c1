"""z-profile samples fall on every multiple of the interval whatever became of the trial there: with a
first stage most titration and swap trials end before an exact energy, moves into a wall without one;
the same in exact runs and in runs that harvest training samples."""
import numpy as np
import pytest

from ph_brush_b200 import Engine, Surrogate, configs

from test_gpu_zhist import host_hist


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["exact", "first stage", "harvest"])
@pytest.mark.parametrize("every", [1, 7, 50])
def test_a_sample_at_every_multiple(mode, every):
    s, p = configs.small_system(seed=12, p_swap=0.2, salt_conc=0.02)
    p.p_disp, p.p_titr, p.disp_max = 0.3, 0.5, 2.0  # (many refused by the first stage or the walls)
    s.capacity += 20
    with Engine(s, p) as e:
        if mode == "first stage":
            e.attach_surrogate(Surrogate(seed=5), threshold=0.0)
        elif mode == "harvest":
            e.harvest(4096)
        e.set_zhist(12, every=every)
        e.run(350)
        h, n = e.zhist()
        assert n == 350 // every
        if mode == "first stage":
            assert e.da_stats()[0]["evaluated"] - e.da_stats()[0]["passed"] > 50
        e.set_zhist(12, every=500)
        e.run(150)  # trial 500 is the next multiple: one sample, the state after it
        h, n = e.zhist()
        assert n == 1 and np.array_equal(h, host_hist(e.state(), p, 12))
