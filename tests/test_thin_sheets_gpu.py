"""Sheets of a few rows step with the column walks: no slower than asked for by flag, the
default form held to the oracle, FP32C with the bits of single steps, alone and in a
batch."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu

STEPS = 7


@pytest.mark.parametrize("source", [False, True])
@pytest.mark.parametrize("shape", [(450, 3, 450), (450, 4, 450), (450, 5, 449), (200, 10, 1015), (450, 11, 450)],
                         ids=lambda s: "x".join(map(str, s)))
def test_values(heat, oracle, cuda_device, shape, source):
    H = heat
    kappa, u0, h, dt = H.inputs_config(0, 19, *shape)
    rhs = 1e-3 * np.random.default_rng(1).random(u0.shape) if source else None
    ref = oracle.steps(u0, kappa, h, dt, STEPS, rhs=rhs)
    with H.Solver(kappa, u0, h, dt, rhs=rhs) as s:
        s.step(STEPS)
        got = s.field()
        assert np.abs(got - ref).max() <= STEPS * 8 * 2.0 ** -52 * (1 + STEPS * 1e-3)
    fields = []
    for flags in (0, H.HEAT_NO_TEMPORAL):
        with H.Solver(kappa, u0, h, dt, rhs=rhs, precision=H.HEAT_FP32C, flags=flags) as s:
            s.step(STEPS)
            fields.append(s.field())
    assert bits_equal(*fields)
    with H.Solver(kappa, u0, h, dt, rhs=rhs) as a, \
            H.Solver(kappa, u0, h, dt, rhs=rhs, precision=H.HEAT_FP32C) as c, H.Batch() as b:
        for s in (a, c):
            b.add(s, STEPS)
        b.run()
        assert bits_equal(a.field(), got) and bits_equal(c.field(), fields[0])


@pytest.mark.parametrize("precision,flag", [("fp64", "HEAT_HWFP64"), ("fp32c", "HEAT_NO_TEMPORAL")])
def test_speed(heat, cuda_device, precision, flag):
    torch, H = cuda_device, heat
    kappa, u0, h, dt = H.inputs_config(0, 3, 2048, 3, 1024)
    stream = torch.cuda.Stream()
    times = []
    for flags in (0, getattr(H, flag)):
        with H.Solver(kappa, u0, h, dt, precision={"fp64": H.HEAT_FP64, "fp32c": H.HEAT_FP32C}[precision],
                      flags=flags, stream=stream.cuda_stream) as s:
            s.step(10)
            best = float("inf")
            for _ in range(5):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record(stream)
                s.step(20)
                b.record(stream)
                b.synchronize()
                best = min(best, a.elapsed_time(b))
            times.append(best)
    assert times[0] <= 1.25 * times[1], times
