"""Batched trials of the plain Monte Carlo kernel: a block evaluates up to 16
consecutive trials against one state and decides them in order.

Every sum of that kernel is formed per probe and per stencil pair in a fixed
order, so a replica's chain must come out bit for bit the same whatever shares
its launch: alone it runs on a cluster of eight blocks and batches of 16; with
more replicas on smaller clusters, one 512-thread block, or (more replicas than
SMs) 256- or 128-thread blocks and batches of 8.  The same chain must follow the
oracle's trial by trial (test_gpu_mc.py) and its energy a full recompute.
"""
import numpy as np
import pytest

from ph_brush_b200 import Engine, configs


def make(seed, order):
    s, p = configs.small_system(seed=seed, order=order, box_xy=13.0, height=13.0, p_swap=0.1, salt_conc=0.02)
    s.capacity += 20
    p.pending_max = 10
    return s, p


def final(s, p, n, threads=256):
    with Engine(s, p) as e:
        e.set_quorum(1.0)
        e.set_tuning(10, threads)
        st = e.run(n)
        R = 1 if not isinstance(s, list) else len(s)
        return st, [e.state(r) for r in range(R)], e.energy()


# replicas: cluster of 4, of 2, none; more replicas than SMs with either block size.  Trials: a
# multiple of no batch length
@pytest.mark.gpu
@pytest.mark.parametrize("order", [4, 5, 6])
@pytest.mark.parametrize("R,threads", [(30, 256), (70, 256), (140, 256), (150, 256), (150, 128)])
def test_a_replica_runs_the_same_in_any_company(order, R, threads):
    n = 203
    solo = [make(50 + k, order) for k in range(2)]
    ref = [final(s, p, n) for s, p in solo]
    reps = [solo[r % 2] for r in range(R)]
    st, states, fresh = final([s for s, _ in reps], [p for _, p in reps], n, threads)
    for r in (0, 1, R - 2, R - 1):
        rs, rst, rf = ref[r % 2]
        for k in rst[0]:
            assert np.array_equal(states[r][k], rst[0][k]), (r, k)
        assert st[r]["energy"] == rs[0]["energy"]
        assert (st[r]["attempted"], st[r]["accepted"]) == (rs[0]["attempted"], rs[0]["accepted"])
        assert sum(st[r]["attempted"]) == n
        assert st[r]["n_anions"] == rs[0]["n_anions"] and st[r]["n_cations"] == rs[0]["n_cations"]


# dense cells (long candidate lists: more than one list window and several full evaluation queues)
# and cell rows that are no multiple of four entries
@pytest.mark.gpu
@pytest.mark.parametrize("cell_cap", [61, 64])
def test_crowded_cells_keep_the_tracked_energy(cell_cap):
    s, p = configs.small_system(seed=9, chains=6, length=14, box_xy=15.0, height=15.0, salt_pairs=500, mesh=(32, 32, 54))
    p.lj_eps = p.lj_eps * 0.0  # ions may crowd
    p.cell_cap = cell_cap
    with Engine(s, p) as e:
        st = e.run(600)[0]
        fresh = e.energy()[0]["total"]
    assert sum(st["accepted"]) > 50
    assert abs(st["energy"] - fresh) <= 1e-6 * abs(fresh) + 1e-3, (st["energy"], fresh)
