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


def test_points_formed_from_the_list_and_in_the_second_walk_agree(heat, cuda_device):
    """A block forms its marked patches from a list where they are few and in a second
    walk where they are many: the same plane of values, once in a grid of few and once in
    one of many, gives the same bits."""
    H = heat
    nx, ny, nz = 34, 18, 40
    kappa, u0, h, dt = H.inputs_config(0, 41, nx, ny, nz)
    rng = np.random.default_rng(2)
    steep = u0 * np.exp2(rng.integers(-60, 1, u0.shape))
    few = u0.copy()
    few[16:23] = steep[16:23]
    results = []
    for u in (few, steep):
        u = u.copy()
        with H.Solver(kappa, u, h, dt) as s:
            s.step(3)
            results.append(s.field()[19])  # depends on planes 16 to 22 alone
    assert np.array_equal(results[0].view(np.uint64), results[1].view(np.uint64))


def test_huge_and_tiny_neighbours(heat, oracle, cuda_device):
    """Points beyond both ends of the patch form's exponents, subnormal ones and ones of
    2^1007 and more among them: a few units of the last place of the largest of the seven
    values, or of the smallest number there is."""
    H = heat
    nx, ny, nz = 37, 21, 26
    kappa, u0, h, dt = H.inputs_config(0, 43, nx, ny, nz)
    rng = np.random.default_rng(8)
    for low, high in ((-1074, -900), (900, 1020), (-1074, 1020)):
        u = u0 * np.ldexp(1.0, rng.integers(low, high, u0.shape)) * rng.choice([-1.0, 1.0], u0.shape)
        with H.Solver(kappa, u, h, dt) as s:
            s.step(1)
            got = s.field()
        ref = oracle.steps(u, kappa, h, dt, 1)
        assert np.all(np.isfinite(ref))
        assert np.all(np.abs(got - ref) <= 5 * 2.0 ** -52 * local_max(u, 1) + 8 * 5e-324)
