"""Conductivities far apart, and steps far below the stable one, in the default FP64
form: heat that seeps into cold places, by weights that are a small part of the fixed
point's range, keeps its relative accuracy.  All values are positive and every weight
is, so nothing cancels and relative errors of a step only add up: at most seven units
of a result of 2^46 units and more, and eight roundings of the oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 12
TOL = STEPS * (7 * 2.0 ** -46 + 8 * 2.0 ** -52)


@pytest.mark.parametrize("source", [False, True])
@pytest.mark.parametrize("low", [1e-3, 1e-6, 1e-9, 1e-13, 1e-30])
@pytest.mark.parametrize("kind", ["cold insulators", "warm", "small steps"])
def test_relative_accuracy(heat, oracle, cuda_device, kind, low, source):
    H = heat
    nx, ny, nz = 36, 35, 23
    rng = np.random.default_rng(6)
    h = 1.0 / (nx - 1)
    dt = 0.9 * h * h / 6.0
    weak = rng.random((nz, ny, nx)) < 0.5
    u0 = rng.random(weak.shape)
    kappa = np.where(weak, low, 1.0)
    if kind == "cold insulators":
        u0[weak] = 0.0
    elif kind == "small steps":
        kappa, dt = np.full(weak.shape, 0.7), dt * low
        u0[nz // 2:] = 0.0
    rhs = low * 1e-3 * rng.random(weak.shape) if source else None
    with H.Solver(kappa, u0, h, dt, rhs=rhs) as s:
        s.step(STEPS)
        got = s.field()
    ref = oracle.steps(u0, kappa, h, dt, STEPS, rhs=rhs)
    assert np.all(np.abs(got - ref) <= TOL * np.abs(ref) + STEPS * 8 * 5e-324)
