"""The full recompute's charge spread with one to four planes to a block (the more replicas, the
more planes): integer sums, so a replica's reciprocal energy is bit for bit what it has in an engine
of four (whose other passes are the same: every mesh of an engine decides on them), whatever the planes per block, with bands that wrap, that are no multiple of the planes,
and that cover every plane of a mesh no deeper than the stencil."""
import pytest

from ph_brush_b200 import Engine, configs


# 48 planes a replica without walls, ~20 with: 1184, 1776 and 2368 planes are the lines to 2, 3 and 4
@pytest.mark.gpu
@pytest.mark.parametrize("order", [4, 5, 6])
@pytest.mark.parametrize("n,walls,nz", [(10, 1, 48), (30, 0, 48), (45, 0, 48), (60, 0, 48), (60, 0, 45), (100, 1, 50), (150, 1, 50), (410, 0, 6)])
def test_planes_per_block(n, walls, nz, order):
    reps = []
    for k in range(4):
        s, p = configs.small_system(seed=80 + k, order=order, mesh=(16, 16 + 2 * (k % 2), nz), salt_pairs=20)
        p.walls = walls
        reps.append((s, p))
    with Engine([s for s, _ in reps], [p for _, p in reps]) as e:
        few = [r["coul_recip"] for r in e.energy()]
    with Engine([reps[k % 4][0] for k in range(n)], [reps[k % 4][1] for k in range(n)]) as e:
        got = [r["coul_recip"] for r in e.energy()]
    assert all(g == few[k % 4] for k, g in enumerate(got))
