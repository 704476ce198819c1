"""The full recompute's charge spread at charges far from one: a single particle of thousands of
units on a mesh point, and six like charges on one, below and above the sum of |q| up to which a
plane is added in two 32-bit halves.  Reciprocal energies against the FP64 oracle at the repository's
tolerance (1e-6 relative / 1e-4 kT)."""
import numpy as np
import pytest

from oracle import pyoracle as O
from ph_brush_b200 import Engine, configs

from test_gpu_energy import close


# an order-p stencil's largest weight, at a mesh point (even orders) or between two (odd): 2/3, 115/192,
# 11/20 per axis; the halves hold 2^11 / weight^3 units on one point: 6912, 9531, 12309
@pytest.mark.gpu
@pytest.mark.parametrize("order", [4, 5, 6])
@pytest.mark.parametrize("total", [6850.0, 6950.0, 8000.0, 9050.0, 20000.0, -8000.0])
@pytest.mark.parametrize("count", [1, 6])
def test_heavy_charges_on_one_mesh_point(order, total, count):
    s, p = configs.small_system(seed=3, order=order)  # mesh spacing 0.75
    at = 6.0 + (0.375 if order % 2 else 0.0)
    add = dict(x=at + 1e-3 * np.arange(count), y=np.full(count, at), z=np.full(count, at), q=np.full(count, total / count))
    for k, v in add.items():
        setattr(s, k, np.concatenate([getattr(s, k), v]).astype(np.float32))
    s.type = np.concatenate([s.type, np.full(count, 3)]).astype(np.int32)
    s.flags = np.concatenate([s.flags, np.full(count, 0x09 if total > 0 else 0x11)]).astype(np.int32)
    s.capacity = s.n + 64
    p.lj_eps = p.lj_eps * 0.0
    with Engine(s, p) as e:
        got = e.energy()[0]["coul_recip"]
        state = e.state()
        e.set_state(state)
        again = e.energy()[0]["coul_recip"]
    ref = O.energy(s, p)["coul_recip"]
    assert close(got, ref), (got, ref)
    assert again == got
