"""Systems without walls (wall_hi <= wall_lo: z periodic): every plane of the mesh holds charge, so the
rebuild's passes and the charge spread run over all of them.  Energies against the FP64 oracle at the
repository's tolerance; the spread's integer sums bit for bit against an engine of four replicas."""
import pytest

from oracle import pyoracle as O
from ph_brush_b200 import Engine, configs

from test_gpu_energy import assert_components, close


def open_system(**kw):
    s, p = configs.small_system(**kw)
    p.wall_lo = p.wall_hi = 0.0
    return s, p


# Stockham depths (one to six stages) and every depth with a register split
@pytest.mark.gpu
@pytest.mark.parametrize("nz", [6, 8, 15, 20, 48, 128, 150, 162, 192, 216, 243, 256, 288, 324, 384, 432])
@pytest.mark.parametrize("nx", [16, 50])
def test_any_depth_without_walls(nz, nx):
    s, p = open_system(seed=nz + nx, mesh=(nx, 18, nz))
    with Engine(s, p) as e:
        assert_components(e.energy()[0], O.energy(s, p))
        st = e.run(400)[0]
        fresh = e.energy()[0]["total"]
    assert sum(st["accepted"]) > 50
    assert close(st["energy"], fresh, 1e-6, 1e-3)


# 48 planes a replica: 1184, 1776 and 2368 planes are the lines to 2, 3 and 4 planes per block
@pytest.mark.gpu
@pytest.mark.parametrize("order", [4, 5, 6])
@pytest.mark.parametrize("n,nz", [(30, 48), (45, 48), (60, 48), (60, 45), (410, 6)])
def test_planes_per_block_without_walls(n, nz, order):
    reps = [open_system(seed=80 + k, order=order, mesh=(16, 16 + 2 * (k % 2), nz), salt_pairs=20) for k in range(4)]
    with Engine([s for s, _ in reps], [p for _, p in reps]) as e:
        few = e.energy()
    for (s, p), c in zip(reps, few):
        assert close(c["coul_recip"], O.energy(s, p)["coul_recip"])
    with Engine([reps[k % 4][0] for k in range(n)], [reps[k % 4][1] for k in range(n)]) as e:
        got = e.energy()
    assert all(g["coul_recip"] == few[k % 4]["coul_recip"] for k, g in enumerate(got))
