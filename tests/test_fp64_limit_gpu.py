"""Time steps at the stability limit: the default FP64 form takes every problem whose
centre weights 1 - sum of the six face weights are 2^-29 and more, right up to sums
that fill its 64 bits, and leaves those without one to the FP64-pipe kernel."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 9
N = 26


def problem(margin, rng, low):
    """A conductivity of (nearly) 1 and a step whose centre weight is about `margin`; the
    weights' low limbs are about `low` of their unit."""
    h = 1.0 / (N - 1)
    weight = (1.0 - margin) / 6.0 / 2.0  # factor * kappa
    weight = np.floor(weight * 2.0 ** 32 - 1) * 2.0 ** -32 + low * 2.0 ** -32
    dt = weight * 2.0 * h * h
    u0 = rng.choice([0.0, 1.0, 1.0 - 2.0 ** -53, 2.0 ** -30, -1.0], (N, N, N))
    return np.ones((N, N, N)), u0, h, dt


@pytest.mark.parametrize("low", [0.0, 0.2, 0.499, 0.501, 0.9])
@pytest.mark.parametrize("margin", [2.0 ** -29, 1e-8, 2.0 ** -24, 1e-7, 2.0 ** -20])
def test_near_the_limit(heat, oracle, cuda_device, margin, low):
    H = heat
    kappa, u0, h, dt = problem(margin, np.random.default_rng(4), low)
    with H.Solver(kappa, u0, h, dt) as s:
        s.step(STEPS)
        got = s.field()
        # it steps with the fixed-point kernel
        assert H.lib().heat_diag_fp64_timeout(s._ctx) == H.HEAT_OK
        assert H.lib().heat_sync(s._ctx) == H.HEAT_ETIMEOUT
    ref = oracle.steps(u0, kappa, h, dt, STEPS)
    # a step's rounding and units, the oracle's seven roundings, relative to the largest value
    assert np.abs(got - ref).max() <= STEPS * 5 * 2.0 ** -52


def test_beyond_the_limit(heat, oracle, cuda_device):
    H = heat
    kappa, u0, h, dt = problem(0.0, np.random.default_rng(4), 2.5)  # centre weights below zero
    with H.Solver(kappa, u0, h, dt) as s:
        s.step(STEPS)
        got = s.field()
        assert H.lib().heat_diag_fp64_timeout(s._ctx) == H.HEAT_ESTATE
    ref = oracle.steps(u0, kappa, h, dt, STEPS)
    assert np.abs(got - ref).max() <= STEPS * 8 * 2.0 ** -52
