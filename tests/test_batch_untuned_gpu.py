"""Tables of the batch engine whose classes are not tuned: odd and even step
counts, with and without a source term, and grids at the edges of the kernels' tiles
(32 x 16 columns FP64; 32 x 20 FP32C alone, whose table walks columns).  Every grid has
the bits it has alone."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu

SHAPES = [(3, 3, 3), (34, 22, 5), (35, 23, 40), (33, 18, 9), (66, 42, 130), (130, 5, 17)]


@pytest.mark.parametrize("forms", ["fp64", "fp32c", "both"])
@pytest.mark.parametrize("steps", [1, 6, 9])
def test_untuned_table_equals_alone(heat, cuda_device, tmp_path, monkeypatch, forms, steps):
    H = heat
    monkeypatch.setenv("HEAT_TUNE_CACHE", str(tmp_path / "none.json"))
    precisions = {"fp64": [H.HEAT_FP64], "fp32c": [H.HEAT_FP32C], "both": [H.HEAT_FP64, H.HEAT_FP32C]}[forms]
    solvers, expected = [], []
    for k, (nx, ny, nz) in enumerate(SHAPES):
        for precision in precisions:
            kappa, u0, h, dt = H.inputs_config(0, k, nx, ny, nz)
            rhs = 1e-3 * np.ones_like(u0) if k % 3 == 2 else None
            with H.Solver(kappa, u0, h, dt, rhs=rhs, precision=precision) as alone:
                alone.step(2 * steps + 1)
                expected.append(alone.field())
            solvers.append(H.Solver(kappa, u0, h, dt, rhs=rhs, precision=precision))
    with H.Batch() as b:
        for n in (steps, steps + 1):  # a second run starts from either buffer
            for s in solvers:
                b.add(s, n)
            b.run()
            for s in solvers:
                b.remove(s)
    for s, ref in zip(solvers, expected):
        assert bits_equal(s.field(), ref)
        s.close()
