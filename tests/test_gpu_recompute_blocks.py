"""The full recompute's partial sums hold what the launch rule asks for at every block size, from the
one of a single replica (a block per few cells) to the few blocks per replica of a thousand: energies
at each size, changed after creation, against the FP64 oracle."""
import pytest

from oracle import pyoracle as O
from ph_brush_b200 import Engine, configs

from test_gpu_energy import assert_components


@pytest.mark.gpu
@pytest.mark.parametrize("R", [1, 7, 150, 1200])
def test_recompute_at_every_block_size(R):
    reps = [configs.small_system(seed=3 + k, box_xy=12.0 + 3 * k) for k in range(2)]
    ref = [O.energy(s, p) for s, p in reps]
    with Engine([reps[r % 2][0] for r in range(R)], [reps[r % 2][1] for r in range(R)]) as e:
        for block in (0, 64, 128, 256, 64):
            e.set_tile_shapes(energy_block=block)
            got = e.energy()
            for r in sorted({0, R // 2, R - 1}):
                assert_components(got[r], ref[r % 2])
