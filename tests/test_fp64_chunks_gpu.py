"""The default FP64 form does not know where a z-chunk or a launch begins: fields of
both signs, steep ones and ones with zeros have the same bits whatever the depth of a
table's tiles, and alone, where patches carry their integers from plane to plane."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu

STEPS = 11


def field(kind, u0, rng):
    nz, ny, nx = u0.shape
    if kind == "signed":
        return np.where(u0 != 0.0, u0 * 2.0 - 1.0, 0.0)
    if kind == "half signed":  # warps with and without negative values, some with both
        u = u0.copy()
        u[:, : ny // 2] *= -1.0
        u[:, :, nx // 2:] = np.abs(u[:, :, nx // 2:])
        return u
    if kind == "steep":
        return u0 * np.exp2(-2.0 * np.arange(nz))[:, None, None] * np.exp2(-1.5 * np.arange(nx))
    if kind == "scattered":
        return u0 * np.exp2(rng.integers(-40, 1, u0.shape)) * rng.choice([-1.0, 1.0], u0.shape)
    if kind == "large":
        return u0 * 1e100 * rng.choice([-1.0, 1.0], u0.shape)
    u = np.zeros_like(u0)
    u[nz // 3: 2 * nz // 3, ny // 3: 2 * ny // 3, nx // 3: 2 * nx // 3] = 1.0
    return u


@pytest.mark.parametrize("source", [False, True])
@pytest.mark.parametrize("kind", ["signed", "half signed", "steep", "scattered", "large", "spot"])
def test_depth_of_tiles_does_not_matter(heat, cuda_device, tmp_path, monkeypatch, kind, source):
    H = heat
    nx, ny, nz = 67, 37, 45
    kappa, u0, h, dt = H.inputs_config(0, 29, nx, ny, nz)
    rng = np.random.default_rng(3)
    u0 = field(kind, u0, rng)
    rhs = rng.uniform(-1e-3, 1e-3, u0.shape) if source else None
    with H.Solver(kappa, u0, h, dt, rhs=rhs) as s:
        s.step(STEPS)
        alone = s.field()
    assert np.all(np.isfinite(alone)) and np.any(alone)
    for depth in (1, 2, 5, 32):
        cache = tmp_path / f"{depth}.json"
        cache.write_text('{"device": "test", "entries": [\n'
                         f' {{"form": 0, "nz_max": 64, "kchunk": {depth}, "glups": 1.0}}\n]}}\n')
        monkeypatch.setenv("HEAT_TUNE_CACHE", str(cache))
        # enough other grids that the table itself does not ask for shorter tiles
        with H.Solver(kappa, u0, h, dt, rhs=rhs) as s, H.Batch() as b:
            others = [H.Solver(kappa, u0, h, dt, rhs=rhs) for _ in range(40 if depth > 2 else 0)]
            for c in [s, *others]:
                b.add(c, STEPS)
            b.run()
            assert bits_equal(s.field(), alone), depth
            for c in others:
                c.close()


def test_either_sign_runs_at_speed(heat, cuda_device):
    """Negative values cost a step little (the code for any sign converts and rounds as
    the other does)."""
    torch, H = cuda_device, heat
    n = 192
    kappa, u0, h, dt = H.inputs_config(0, 3, n, n, n)
    stream = torch.cuda.Stream()
    times = []
    sine = np.sin(np.arange(n) * (4 * np.pi / (n - 1)))
    for u in (u0, -u0, u0 * sine[:, None, None]):
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
    assert max(times[1:]) <= 1.33 * times[0], times
