"""Tables that hold default FP64 grids (four tensor maps each) and two-step FP32C
grids (seven) side by side, rebuilt while launches and uploads run: every grid has
the bits it has alone."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu

FORMS, CLASSES = range(5), (64, 128, 256, 384)


@pytest.fixture
def H(heat, cuda_device, tmp_path, monkeypatch):
    """Tuned classes with two FP32C steps per launch, so that those grids use maps."""
    lines = [f' {{"form": {f}, "nz_max": {c}, "kchunk": 16, "rows": 1, "minb": 3, "depth": 2, "glups": 1.0}}'
             for f in FORMS for c in CLASSES]
    cache = tmp_path / "tune.json"
    cache.write_text('{"device": "test", "entries": [\n' + ",\n".join(lines) + "\n]}\n")
    monkeypatch.setenv("HEAT_TUNE_CACHE", str(cache))
    return heat


def shape(q):
    return 18 + 7 * (q % 9), 20 + 3 * (q % 11), 12 + 5 * (q % 8)


def alone(H, q, steps, precision):
    kappa, u0, h, dt = H.inputs_config(0, q, *shape(q))
    with H.Solver(kappa, u0, h, dt, precision=precision) as s:
        s.step(steps)
        return s.field()


def test_batch_whose_members_come_and_go(H):
    waiting = [(q, 3 + q % 13, H.HEAT_FP32C if q % 3 else H.HEAT_FP64) for q in range(48)]
    expected = {q: alone(H, q, n, p) for q, n, p in waiting}
    live, left = {}, list(waiting)
    with H.Batch() as b:
        while left or live:
            while left and len(live) < 12:
                q, n, p = left.pop()
                kappa, u0, h, dt = H.inputs_config(0, q, *shape(q))
                live[q] = H.Solver(kappa, u0, h, dt, precision=p)
                b.add(live[q], n)
            b.run(2)
            for q in [q for q, s in live.items() if b.pending(s) == 0]:
                s = live.pop(q)
                assert bits_equal(s.field(), expected[q]), q
                b.remove(s)
                s.close()


def test_server_requests_of_both_kinds(H):
    reqs = [(q, 5 + q % 29, H.HEAT_FP32C if q % 2 else H.HEAT_FP64) for q in range(80)]
    outs = [np.empty(shape(q)[::-1]) for q, _, _ in reqs]
    with H.Server(8 << 30, tick_steps=4, prep_threads=4) as srv:
        for (q, n, p), o in zip(reqs, outs):
            srv.submit(*shape(q), steps=n, seed=q, precision=p, field_out=o)
        srv.wait_idle()
        assert all(r["status"] == 0 for r in srv.poll())
    for (q, n, p), o in zip(reqs, outs):
        assert bits_equal(alone(H, q, n, p), o), q
