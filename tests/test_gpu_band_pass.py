"""The rebuild's z pass over a leading band: every split of every listed depth, with the band
wrapping below plane 0 (walls at the bottom), ending on a split's last admitted plane, and where it
does not fit (walls higher up) and the general pass takes it.  Energies against the FP64 oracle at
the repository's tolerance, and trial energies against the shared-memory pass (FP32 potentials of
one charge mesh: 1e-5 relative, 1e-4 kT)."""
import numpy as np
import pytest

from oracle import pyoracle as O
from ph_brush_b200 import Engine, configs

from test_gpu_energy import assert_components, close

SPLITS = {48: (1, 10), 128: (2, 11), 162: (3, 12), 192: (4, 13), 216: (5, 14), 243: (6, 15), 256: (7,), 288: (8, 16),
          384: (9, 17, 18)}


@pytest.mark.gpu
@pytest.mark.parametrize("nz", sorted(SPLITS))
@pytest.mark.parametrize("order,lift", [(5, 0.0), (4, 0.0), (6, 0.0), (5, 1.5), (5, 12.0)])
def test_band_pass(nz, order, lift):
    s, p = configs.small_system(seed=nz + order, order=order, mesh=(16, 18, nz))
    s.z = (s.z + np.float32(lift)).astype(np.float32)
    p.wall_lo += lift
    p.wall_hi += lift
    ref = O.energy(s, p)
    i = int(np.flatnonzero(s.q != 0)[-1])
    moves = [[dict(index=i, x=float(s.x[i]), y=float(s.y[i]), z=float(z), q=float(s.q[i]), type=int(s.type[i]))]
             for z in np.linspace(p.wall_lo + 0.01, p.wall_hi - 0.01, 24)]
    dE = {}
    for v in (0,) + SPLITS[nz]:
        with Engine(s, p) as e:
            e.set_tile_shapes(zpass=v)
            assert_components(e.energy()[0], ref)
            dE[v] = [d["coul_recip"] for d in e.delta_energy_components(moves)]
    for v in SPLITS[nz]:
        assert all(close(a, b, 1e-5, 1e-4) for a, b in zip(dE[v], dE[0]))


@pytest.mark.gpu
@pytest.mark.parametrize("nz", [5, 6, 8, 15, 20, 150, 324, 432])
@pytest.mark.parametrize("nx", [16, 36, 50])
def test_any_depth(nz, nx):
    """The Stockham pass: one to six stages of radices 2 to 5, column counts that do not fill a
    block's sixteen, with walls and without (every plane holds charge)."""
    for walls in (1, 0):
        s, p = configs.small_system(seed=nz + nx, mesh=(nx, 18, nz))
        p.walls = walls
        ref = O.energy(s, p)
        with Engine(s, p) as e:
            if e.tuning()["zpass"]:
                e.set_tile_shapes(zpass=0)
            assert_components(e.energy()[0], ref)
            st = e.run(400)[0]
            fresh = e.energy()[0]["total"]
            assert close(st["energy"], fresh, 1e-6, 1e-3)
