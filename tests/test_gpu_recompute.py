"""The full recompute where its kernels take another turn: cells of more particles than one warp
holds at a time, candidate lists longer than one chunk, and charge planes that more charges reach
than the split 32-bit sums can hold.  Energies against the FP64 oracle, at the repository's
tolerance (1e-6 relative / 1e-4 kT per component)."""
import numpy as np
import pytest

from oracle import pyoracle as O
from ph_brush_b200 import Engine, configs

from test_gpu_energy import assert_components


def crowd(salt_pairs, order=5, layer=None, seed=3):
    """A small brush with many ions that do not repel (LJ off); layer: all ions in a sheet of that depth."""
    s, p = configs.small_system(seed=seed, box_xy=12.0, height=12.0, salt_pairs=4, order=order)
    rng = np.random.default_rng(seed)
    n = 2 * salt_pairs
    z = rng.uniform(0.5, 11.5, n) if layer is None else rng.uniform(6.0, 6.0 + layer, n)
    add = dict(x=rng.uniform(0, 12, n), y=rng.uniform(0, 12, n), z=z, q=np.tile([1.0, -1.0], salt_pairs))
    for k, v in add.items():
        setattr(s, k, np.concatenate([getattr(s, k), v]).astype(np.float32))
    s.type = np.concatenate([s.type, np.tile([3, 2], salt_pairs)]).astype(np.int32)
    s.flags = np.concatenate([s.flags, np.tile([0x09, 0x11], salt_pairs)]).astype(np.int32)
    s.capacity = s.n + 64
    p.lj_eps = p.lj_eps * 0.0
    p.cell_cap = 4096
    return s, p


# pairs of ions: about 3, 12 and 40 particles in a cell (one own block, several chunks, several own blocks)
@pytest.mark.gpu
@pytest.mark.parametrize("block", [0, 64, 128, 256])
@pytest.mark.parametrize("pairs", [100, 380, 1300])
def test_crowded_cells(pairs, block):
    s, p = crowd(pairs)
    with Engine(s, p) as e:
        e.set_tile_shapes(energy_block=block)
        got = e.energy()[0]
    assert_components(got, O.energy(s, p))


# 4000 and 4400 charges in one sheet: below and above what a plane's 32-bit halves are allowed
@pytest.mark.gpu
@pytest.mark.parametrize("order", [4, 5, 6])
@pytest.mark.parametrize("pairs", [1950, 2200])
def test_crowded_planes(pairs, order):
    s, p = crowd(pairs, order=order, layer=0.05)
    with Engine(s, p) as e:
        got = e.energy()[0]
    ref = O.energy(s, p)
    assert abs(got["coul_recip"] - ref["coul_recip"]) <= 1e-6 * abs(ref["coul_recip"]) + 1e-4
