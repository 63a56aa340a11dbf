"""Fields that are zero, of either sign, in most places: hot spots, single points,
zeros up to a wall, with and without a source term, over tile and chunk edges.  Zeros
all around stay exactly +0.0; everything else is held to the oracle within 12 steps of
five units of the last place (a step's rounding, a unit of the fixed point, the
oracle's seven roundings) of the largest value within 12 points."""
from __future__ import annotations

import numpy as np
import pytest

from test_fp64_fx_gpu import STEPS, TOL, local_max

pytestmark = pytest.mark.gpu

SHAPES = [(5, 6, 7), (34, 19, 40), (66, 35, 70)]


def cold(kind, shape, rng):
    nx, ny, nz = shape
    u = np.zeros((nz, ny, nx))
    if kind == "point":
        u[nz // 2, ny // 2, nx // 2] = 1.0
    elif kind == "signed zeros":
        u = np.where(rng.random(u.shape) < 0.5, 0.0, -0.0)
        u[nz // 2, ny // 2, 1] = -3.0
    elif kind == "spots":
        u[rng.random(u.shape) < 0.002] = 1.0
        u[rng.random(u.shape) < 0.002] = -1e-3
    elif kind == "half":
        u[:, :, nx // 2:] = rng.random((nz, ny, nx - nx // 2))
    elif kind == "subnormal":
        u[nz // 3:, 1:-1, 1:-1] = 5e-324
    return u


@pytest.mark.parametrize("source", [False, True])
@pytest.mark.parametrize("kind", ["zero", "point", "signed zeros", "spots", "half", "subnormal"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_against_the_oracle(heat, oracle, cuda_device, shape, kind, source):
    H = heat
    nx, ny, nz = shape
    rng = np.random.default_rng(11)
    kappa, _, h, dt = H.inputs_config(0, 17, nx, ny, nz)
    u0 = cold(kind, shape, rng)
    rhs = None
    if source:
        rhs = np.zeros_like(u0)
        rhs[nz // 2, ny // 2, 1:3] = 1e-3
    with H.Solver(kappa, u0, h, dt, rhs=rhs) as s:
        s.step(STEPS)
        got = s.field()
    ref = oracle.steps(u0, kappa, h, dt, STEPS, rhs=rhs)
    top = local_max(u0) + (STEPS * local_max(rhs) if source else 0)
    assert np.all(np.abs(got - ref) <= TOL * top + STEPS * 8 * 5e-324)
    still = local_max(u0, 2 * STEPS) + (local_max(rhs, 2 * STEPS) if source else 0) == 0
    inside = np.zeros(u0.shape, bool)
    inside[1:-1, 1:-1, 1:-1] = True
    assert not np.any(np.signbit(got[still & inside])) and not np.any(got[still])


def test_zero_regions_run_at_speed(heat, cuda_device):
    """A step over zeros moves its 24 bytes a point and forms nothing: it does not take longer
    than one over a field of values."""
    torch, H = cuda_device, heat
    n = 192
    kappa, u0, h, dt = H.inputs_config(0, 3, n, n, n)
    stream = torch.cuda.Stream()
    times = []
    for u in (u0, np.zeros_like(u0)):
        with H.Solver(kappa, u, h, dt, stream=stream.cuda_stream) as s:
            s.step(20)
            best = float("inf")
            for _ in range(5):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record(stream)
                s.step(40)
                b.record(stream)
                b.synchronize()
                best = min(best, a.elapsed_time(b))
            times.append(best)
    assert times[1] <= 2 * times[0], times
