"""The leading-band z pass computes the operations of the general register pass with their roundings:
beside a replica without walls, whose band covers every plane, an engine takes the general pass for
all, and a replica's reciprocal energy and its trials' must come out bit for bit the same."""
import numpy as np
import pytest

from ph_brush_b200 import Engine, configs

from test_gpu_band_pass import SPLITS


@pytest.mark.gpu
@pytest.mark.parametrize("order", [4, 5, 6])
@pytest.mark.parametrize("nz", sorted(SPLITS))
def test_band_pass_equals_the_general_pass(nz, order):
    s, p = configs.small_system(seed=nz + order, order=order, mesh=(16, 18, nz))
    o, q = configs.small_system(seed=1, order=order, mesh=(16, 18, nz))
    q.wall_lo = q.wall_hi = 0.0
    i = int(np.flatnonzero(s.q != 0)[-1])
    moves = [[dict(index=i, x=float(s.x[i]), y=float(s.y[i]), z=float(z), q=float(s.q[i]), type=int(s.type[i]))]
             for z in np.linspace(p.wall_lo + 0.01, p.wall_hi - 0.01, 24)]
    for v in SPLITS[nz]:
        out = []
        for reps in ([(s, p)], [(s, p), (o, q)]):
            with Engine([a for a, _ in reps], [b for _, b in reps]) as e:
                e.set_tile_shapes(zpass=v)
                out.append([e.energy()[0]["coul_recip"]] + [d["coul_recip"] for d in e.delta_energy_components(moves)])
        assert out[0] == out[1], (v, [k for k in range(25) if out[0][k] != out[1][k]])
