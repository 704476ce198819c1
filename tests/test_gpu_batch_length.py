"""A block chooses how many trials it draws at a time by how often accepted ones cut its recent batches
short: with titrations and ion swaps, which change the lists that proposals draw from, that is a few,
with displacements up to sixteen.  The chain must not depend on it: alone (a cluster of eight blocks),
in company (smaller clusters, one block, blocks of 256 and 128 threads) and in one call or many it
comes out bit for bit the same, and follows the oracle's one-at-a-time trials."""
import numpy as np
import pytest

from ph_brush_b200 import Engine, configs

from test_gpu_mc import replay_check

MIXES = {"titrations": (0.0, 1.0, 0.0), "swaps": (0.3, 0.2, 0.5), "then displacements": (0.9, 0.1, 0.0)}


def system(mix, seed=6):
    s, p = configs.small_system(seed=seed, salt_pairs=8, salt_conc=0.02)
    s.capacity += 60
    p.p_disp, p.p_titr, p.p_swap = MIXES[mix]
    p.pending_max = 24
    return s, p


def chain(R, calls, mix, threads=256):
    s, p = system(mix)
    with Engine([s] * R, [p] * R) as e:
        e.set_quorum(1.0)
        e.set_tuning(24, threads)
        for n in calls:
            st = e.run(n)
        return e.state(R - 1), st[R - 1]["energy"], e.energy()[R - 1]


@pytest.mark.gpu
@pytest.mark.parametrize("mix", sorted(MIXES))
def test_chains_do_not_depend_on_the_batches(mix):
    ref = chain(1, (307,), mix)
    for R, calls, threads in ((1, (1, 2, 101, 203), 256), (30, (307,), 256), (70, (307,), 256), (140, (300, 7), 256),
                              (150, (307,), 256), (150, (100, 207), 128)):
        got = chain(R, calls, mix, threads)
        assert all(np.array_equal(got[0][k], ref[0][k]) for k in ref[0]), (R, calls)
        assert got[2] == ref[2]
        if len(calls) == 1:  # (the rebuild at a call's end changes later trials' last bits)
            assert got[1] == ref[1]


@pytest.mark.gpu
@pytest.mark.parametrize("mix", ["titrations", "swaps"])
def test_short_batches_follow_the_oracle(mix):
    s, p = system(mix)
    st, acc = replay_check(s, p, 300)
    assert acc.sum() > 60
