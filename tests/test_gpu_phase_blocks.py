"""The reference's phases on either block size of their kernel (512 threads while every job has an SM
to itself, 128 beyond) and through many short launches: the same draws and decisions as one job alone.
The sums differ only in the order of FP64 additions (~1e-12 relative), far below the float rounding of
the energies that decide, so counts and the generator's state must be equal and the float energies
within two units in the last place.  After rejected four-point moves the kept charge mesh must still be
that of the present charges (reciprocal energies of probe trials bit for bit those of a fresh upload)."""
import numpy as np
import pytest

from ph_brush_b200 import Engine

from test_gc_phase import CL, NHN, NHP, W, gc_setup, mt_seeded


def p2_job(job, mt, replica=0, attempts=60):
    pools = {k: job[k] for k in ("nh_p", "nh_n", "w", "cl")}
    return dict(replica=replica, nh_n_type=NHN, nh_p_type=NHP, w_type=W, cl_type=CL, q_nh_p=1.0, q_cl=-1.0, beta=1.0,
                max_attempts=attempts, patience=1 << 20, energy_interval=50, z_cut=5.0, mt_state=mt, **pools)


@pytest.mark.gpu
@pytest.mark.parametrize("jobs", [148, 149, 160])
def test_phase2_on_either_block_size(jobs):
    s, p, job = gc_setup()
    mt1 = mt_seeded(5)
    with Engine(s, p) as e:
        (one, _), = e.phase2([p2_job(job, mt1)])
        t1 = e.state()["type"]
    mts = [mt_seeded(5) for _ in range(jobs)]
    with Engine([s] * jobs, [p] * jobs) as e:
        out = e.phase2([p2_job(job, mts[k], k) for k in range(jobs)])
        for k in (0, jobs - 1):
            res = out[k][0]
            assert (res["attempted"], res["accepted"]) == (one["attempted"], one["accepted"])
            assert abs(res["E"] - one["E"]) <= 2 * np.spacing(np.float32(abs(one["E"])))
            assert np.array_equal(mts[k], mt1) and np.array_equal(e.state(k)["type"], t1)


@pytest.mark.gpu
@pytest.mark.parametrize("pend", [6, 7, 48])
def test_rejected_four_point_moves_leave_no_trace(pend):
    s, p, job = gc_setup()
    mt = mt_seeded(11)
    with Engine(s, p) as a, Engine(s, p) as b:
        a.set_tuning(pend, 256)
        (res, _), = a.phase2([p2_job(job, mt, attempts=200)])
        assert 0 < res["accepted"] < res["attempted"] == 200
        cur = a.state()
        b.set_state(cur)
        live = np.flatnonzero(((cur["flags"] & 4) == 0) & (cur["q"] != 0.0))[:24]
        trials = [[dict(index=i, x=(cur["x"][i] + 0.1) % s.box[0], y=cur["y"][i], z=cur["z"][i], q=cur["q"][i],
                        type=cur["type"][i])] for i in live]
        ra = [c["coul_recip"] for c in a.delta_energy_components(trials)]
        rb = [c["coul_recip"] for c in b.delta_energy_components(trials)]
        assert ra == rb
