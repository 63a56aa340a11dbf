"""The bit-exact kernels (context form and heat_update) where they can go wrong:
rows that start and end inside a warp, grids narrower than one, values and
conductivities outside the range their integer arithmetic covers, zeros of both
signs, subnormals, operands far apart, exact ties and cancellations.  Every result
has the oracle's bits."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu

STEPS = 5


@pytest.fixture(scope="module")
def H(heat, cuda_device):
    return heat


def spread(rng, shape, low, high):
    """Uniform significands, exponents from low to high - 1, either sign."""
    return rng.uniform(1, 2, shape) * np.exp2(rng.integers(low, high, shape)) * rng.choice([-1, 1], shape)


def problem(kind, H, shape, source):
    nx, ny, nz = shape
    kappa, u0, h, dt = H.inputs_config(0, 31, nx, ny, nz)
    rng = np.random.default_rng(7)
    inside = np.zeros(u0.shape, bool)
    inside[1:-1, 1:-1, 1:-1] = True
    rhs = rng.uniform(-1e-3, 1e-3, u0.shape) if source else None
    u = {
        "plain": lambda: u0,
        "signed": lambda: u0 - 0.5,
        "zeros": lambda: rng.choice([0.0, -0.0, 1.0, -1.0], u0.shape),
        "near": lambda: 1.0 + rng.integers(-3, 4, u0.shape) * 2.0 ** -52,  # cancels to a few bits
        "short": lambda: rng.integers(-9, 10, u0.shape) * 2.0 ** rng.integers(-53, 1, u0.shape),  # ties
        "far": lambda: spread(rng, u0.shape, -40, 41),
        "small": lambda: spread(rng, u0.shape, -1060, -1000),  # down to subnormals
        "large": lambda: spread(rng, u0.shape, 600, 720),
        "soft": lambda: u0, "hard": lambda: u0, "mixed": lambda: u0, "powers": lambda: u0,
    }[kind]()
    if kind in ("soft", "hard"):  # conductivities outside [2^-200, 2^200]
        e = -400.0 if kind == "soft" else 400.0
        kappa, dt = kappa * 2.0 ** e, dt * 2.0 ** -e
    if kind == "mixed":  # sums of two conductivities far apart, and zeros
        kappa = kappa * np.exp2(-rng.integers(0, 70, kappa.shape).astype(float))
        kappa[rng.random(kappa.shape) < 0.05] = 0.0
    if kind == "powers":  # sums that round up to a power of two, and ties
        kappa = rng.choice([1.0 - 2.0 ** -53, 1.0, 2.0 ** -53, 3 * 2.0 ** -54, 2.0 ** -60], kappa.shape)
        dt = 0.1 * h * h
    return np.where(inside, u, 0.0 if kind != "zeros" else u), kappa, rhs, h, dt


SHAPES = [(3, 3, 3), (4, 41, 5), (18, 9, 7), (32, 5, 40), (33, 8, 4), (63, 14, 6), (130, 23, 35)]


@pytest.mark.parametrize("kind", ["plain", "signed", "zeros", "near", "short", "far", "small", "large",
                                  "soft", "hard", "mixed", "powers"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_oracle_bits(H, oracle, cuda_device, shape, kind):
    torch = cuda_device
    nx, ny, nz = shape
    for source in (False, True):
        u0, kappa, rhs, h, dt = problem(kind, H, shape, source)
        ref = oracle.steps(u0, kappa, h, dt, STEPS, rhs=rhs)
        assert np.all(np.isfinite(ref))
        with H.Solver(kappa, u0, h, dt, rhs=rhs, flags=H.HEAT_BITEXACT) as s:
            s.step(STEPS)
            assert bits_equal(s.field(), ref)
        a, k = torch.from_numpy(u0).cuda(), torch.from_numpy(kappa).cuda()
        b, r = a.clone(), None if rhs is None else torch.from_numpy(rhs).cuda()
        for _ in range(STEPS):
            H.check(H.lib().heat_update(b.data_ptr(), a.data_ptr(), None if r is None else r.data_ptr(),
                                        k.data_ptr(), nz, ny, nx, oracle.factor(h, dt), 0), "heat_update")
            a, b = b, a
        torch.cuda.synchronize()
        assert bits_equal(a.cpu().numpy(), ref)
