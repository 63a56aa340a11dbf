"""The default FP64 form's fixed-point kernel where it can go wrong: edges of
its 32 x 16-column tiles and of its z-chunks, signed data, magnitudes near both
ends of the exponent range and across the bounds of the shared scale, zeros
beside values, and a source term far smaller or far larger than the field.

Tolerance: a step rounds once (1/2 ulp) and adds at most about one more ulp of the
largest of the seven values (a unit of the fixed-point scale is at most 1/4 ulp
inside its bounds); the oracle's seven products and sums add up to 7/2 ulps.
Without a source term a step's result is a convex combination of those values, so
errors relative to the field's local maximum only add up: 12 steps stay below
12 * 5 * 2^-52 = 1.4e-14 of the largest value within 12 points."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu

STEPS = 12
TOL = STEPS * 5 * 2.0 ** -52


@pytest.fixture(scope="module")
def H(heat, cuda_device):
    return heat


def local_max(a, r=STEPS):
    """max |a| over a (2r + 1)-wide box around each point."""
    a = np.abs(a)
    for ax in range(3):
        p = np.pad(a, [(r, r) if k == ax else (0, 0) for k in range(3)])
        a = np.max([np.roll(p, s, axis=ax) for s in range(-r, r + 1)], axis=0)
        a = np.take(a, range(r, r + a.shape[ax] - 2 * r), axis=ax)
    return a


def field(kind, u0, rng):
    inside = u0 != 0.0
    if kind == "signed":
        return np.where(inside, u0 * 2.0 - 1.0, 0.0)
    if kind == "huge":       # scales above 2^60, where values are aligned on the integer pipes
        return u0 * 1e200
    if kind == "tiny":       # near the smallest scale the fixed-point form takes
        return u0 * 2.0 ** -900 * np.exp2(rng.integers(-8, 9, u0.shape))
    if kind == "range":      # patches on both sides of the shared scale's bounds
        return u0 * np.exp2(rng.integers(-9, 1, u0.shape))
    if kind == "holes":
        return np.where(rng.random(u0.shape) < 0.3, 0.0, u0)
    return u0


SHAPES = [(3, 3, 3), (31, 17, 5), (32, 18, 9), (33, 19, 40), (34, 20, 7), (65, 33, 21), (66, 34, 75)]


@pytest.mark.parametrize("kind", ["plain", "signed", "huge", "tiny", "range", "holes"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_against_the_oracle(H, oracle, shape, kind):
    nx, ny, nz = shape
    kappa, u0, h, dt = H.inputs_config(0, 31, nx, ny, nz)
    u0 = field(kind, u0, np.random.default_rng(7))
    with H.Solver(kappa, u0, h, dt) as s:
        s.step(STEPS)
        got = s.field()
    ref = oracle.steps(u0, kappa, h, dt, STEPS)
    assert np.all(np.abs(got - ref) <= TOL * local_max(u0))


@pytest.mark.parametrize("scale", [1e-30, 1.0, 1e30])
def test_source_term_of_any_size(H, oracle, scale):
    kappa, u0, h, dt = H.inputs_config(0, 13, 35, 21, 18)
    rhs = np.random.default_rng(5).uniform(-scale, scale, u0.shape)
    with H.Solver(kappa, u0, h, dt, rhs=rhs) as s:
        s.step(STEPS)
        got = s.field()
    ref = oracle.steps(u0, kappa, h, dt, STEPS, rhs=rhs)
    # the field grows by at most `scale` a step
    assert np.all(np.abs(got - ref) <= TOL * (np.abs(u0).max() + STEPS * scale))


@pytest.mark.parametrize("value", [1.0 / 3.0, -7e-200, 1e250])
def test_a_constant_field_stays_constant(H, value):
    kappa, u0, h, dt = H.inputs_config(0, 3, 40, 23, 19)
    u0 = np.full_like(u0, value)
    with H.Solver(kappa, u0, h, dt) as s:
        s.step(25)
        assert bits_equal(s.field(), u0)


def test_many_short_requests_of_one_form(H):
    """The batch's tables are rebuilt while its launches follow each other without
    a pause: every request still gets its own grid's result."""
    shapes = [(18 + 7 * (q % 5), 20 + 3 * (q % 7), 12 + 5 * (q % 6)) for q in range(90)]
    outs = [np.empty(s[::-1]) for s in shapes]
    with H.Server(8 << 30, tick_steps=4, prep_threads=4) as srv:
        for q, (s, o) in enumerate(zip(shapes, outs)):
            srv.submit(*s, steps=5 + q % 37, seed=q, field_out=o)
        srv.wait_idle()
        assert all(r["status"] == 0 for r in srv.poll())
    for q in range(0, 90, 7):
        kappa, u0, h, dt = H.inputs_config(0, q, *shapes[q])
        with H.Solver(kappa, u0, h, dt) as a:
            a.step(5 + q % 37)
            assert bits_equal(a.field(), outs[q]), q
