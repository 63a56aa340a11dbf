"""The default FP64 form does not drift: with a constant conductivity every face drops
the same fraction of its weight's low limb, so what is dropped must be of either sign.

The conductivity is the one whose low limb is largest (just under or over half of the
high limb's unit, 2^-32), where one-signed drops add up to three units of the fixed
point a step, 300 times 3 / 2^59 = 1.6e-15 of a value near its scale.  Unbiased ones
leave less than a quarter of a unit a step on average over the points."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 300


@pytest.mark.parametrize("low", [0.4999, 0.5001])
def test_mean_error_of_a_long_run(heat, cuda_device, low):
    H = heat
    n, dt = 18, 1e-4
    h = 1.0 / (n - 1)
    weight = (np.floor(0.05 * 2.0 ** 32) + low) * 2.0 ** -32  # factor * kappa
    kappa = np.full((n, n, n), weight * 2.0 * h * h / dt)
    u0 = np.zeros((n, n, n))
    u0[1:-1, 1:-1, 1:-1] = np.random.default_rng(1).random((n - 2,) * 3)
    with H.Solver(kappa, u0, h, dt) as s:
        s.step(STEPS)
        got = s.field()
    long = np.longdouble
    w = long(dt / h / h / 2.0) * (long(kappa[0, 0, 0]) * 2)
    u = u0.astype(long)
    for _ in range(STEPS):
        c = u[1:-1, 1:-1, 1:-1]
        near = (u[2:, 1:-1, 1:-1] + u[:-2, 1:-1, 1:-1] + u[1:-1, 2:, 1:-1] + u[1:-1, :-2, 1:-1]
                + u[1:-1, 1:-1, 2:] + u[1:-1, 1:-1, :-2])
        u[1:-1, 1:-1, 1:-1] = c + w * (near - 6 * c)
    inside = np.s_[1:-1, 1:-1, 1:-1]
    error = ((got[inside].astype(long) - u[inside]) / u[inside]).astype(float)
    assert abs(error.mean()) <= STEPS * 0.25 * 2.0 ** -59
