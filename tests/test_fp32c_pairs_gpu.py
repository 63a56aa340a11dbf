"""The two-step FP32C tile (32 x 20 columns, points in packed pairs) at its edges:
one column or row short of, at and past a tile, the last pair half outside the grid,
z-extents around a chunk, signed values and zeros.  Its bits are those of two
single steps."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [3, 33, 34, 35, 67])
@pytest.mark.parametrize("ny,nz", [(21, 4), (22, 131), (23, 3), (42, 17), (43, 40)])
def test_tile_edges(heat, cuda_device, nx, ny, nz):
    H = heat
    kappa, u0, h, dt = H.inputs_config(0, nx, nx, ny, nz)
    rng = np.random.default_rng(ny)
    u0 = np.where(rng.random(u0.shape) < 0.1, 0.0, u0 * rng.choice([-1.0, 1.0], u0.shape))
    with H.Solver(kappa, u0, h, dt, precision=H.HEAT_FP32C) as a, \
            H.Solver(kappa, u0, h, dt, precision=H.HEAT_FP32C, flags=H.HEAT_NO_TEMPORAL) as b:
        for steps in (2, 5):
            a.step(steps)
            b.step(steps)
            assert bits_equal(a.field(), b.field())
