"""The autotuner's candidates that launch the same code share one timing, so that noise does not
choose among them, and the first of them is kept: the block size in force where every replica takes
blocks of 512 threads, the pair pass's default shape for plain runs, its width alone for runs with a
first stage, 256 threads of a recompute block under both of their names."""
import pytest

from ph_brush_b200 import Engine, configs
from ph_brush_b200.engine import Surrogate

SHAPES = [(2, 2), (8, 2), (2, 3), (2, 4), (2, 21), (4, 21)]


def tuned(R, threads, surrogate):
    reps = [configs.small_system(seed=60 + k) for k in range(R)]
    with Engine([s for s, _ in reps], [p for _, p in reps]) as e:
        e.set_tuning(16, threads)
        if surrogate:
            e.attach_surrogate(Surrogate(seed=5), threshold=0.0)
        res = e.autotune(64)
        st = e.run(200)
        fresh = e.energy()
        for a, b in zip(st, fresh):
            assert abs(a["energy"] - b["total"]) <= 1e-6 * abs(b["total"]) + 1e-3
        return res, e.tuning()


@pytest.mark.gpu
@pytest.mark.parametrize("R,threads,surrogate", [(2, 128, False), (2, 256, False), (2, 128, True), (150, 256, False)])
def test_same_code_shares_one_timing(R, threads, surrogate):
    res, t = tuned(R, threads, surrogate)
    blocks = {r["energy_block"]: r["recompute_us"] for r in res if r["recompute_us"] > 0}
    assert set(blocks) == {0, 64, 128, 256} and blocks[0] == blocks[256] and t["energy_block"] != 256
    runs = [r for r in res if r["us_per_trial"] > 0]  # 8 capacities x 2 block sizes, 6 shapes, the first stage on and off
    assert len(runs) == 22 + 2 * surrogate
    grid = {(r["pending_max"], r["threads"]): r["us_per_trial"] for r in runs[:16]}
    pends = sorted({pm for pm, _ in grid})
    assert len(grid) == 16 and len(pends) == 8
    same = sum(grid[pm, 128] == grid[pm, 256] for pm in pends)
    assert same == 8 and t["threads"] == threads if R == 2 else same < 8
    shape = {(r["cand_round"], r["g_rows"]): r["us_per_trial"] for r in runs[16:22]}
    assert set(shape) == set(SHAPES)
    best = min(grid.values())
    assert shape[2, 2] == shape[2, 3] == shape[2, 4] == shape[2, 21] and shape[4, 21] == best
    if surrogate:
        assert (t["cand_round"], t["g_rows"]) in [(4, 2), (2, 2), (8, 2)] and shape[8, 2] != shape[2, 2]
    else:
        assert set(shape.values()) == {best} and (t["cand_round"], t["g_rows"]) == (4, 2)
