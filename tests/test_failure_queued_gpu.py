"""Work queued behind a launch whose bounded wait ran out leaves at once: nothing is
written, the status surfaces once at the next synchronising call, and the context
steps on from where it stood.  (The flag is set by the product kernels launched with
a wait limit of 0; no wait of these tests runs out otherwise.)"""
from __future__ import annotations

import ctypes as C

import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu


@pytest.fixture
def H(heat, cuda_device, tmp_path, monkeypatch):
    """Tuned classes with two FP32C steps per launch, so that tables use the TMA kernels."""
    cache = tmp_path / "tune.json"
    cache.write_text('{"device": "test", "entries": [\n'
                     ' {"form": 3, "nz_max": 64, "kchunk": 16, "rows": 1, "minb": 3, "depth": 2, "glups": 1.0}\n]}\n')
    monkeypatch.setenv("HEAT_TUNE_CACHE", str(cache))
    return heat


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("batched", [False, True])
def test_steps_behind_a_failure_write_nothing(H, precision, batched):
    lib = H.lib()
    prec, fail = {"fp64": (H.HEAT_FP64, lib.heat_diag_fp64_timeout),
                  "fp32c": (H.HEAT_FP32C, lib.heat_diag_fp32c_timeout)}[precision]
    kappa, u0, h, dt = H.inputs_config(0, 7, 70, 45, 38)
    with H.Solver(kappa, u0, h, dt, precision=prec) as s, H.Batch() as b:
        s.step(4)
        before = s.field()
        assert fail(s._ctx) == H.HEAT_OK
        if batched:
            b.add(s, 40)
            n = C.c_longlong()
            assert lib.heat_batch_run(b._b, -1, C.byref(n)) == H.HEAT_ETIMEOUT and n.value == 40
            b.remove(s)
        else:
            s.step(40)  # an even number of swaps: the current buffer is the one read before
            assert lib.heat_sync(s._ctx) == H.HEAT_ETIMEOUT
        assert lib.heat_sync(s._ctx) == H.HEAT_OK
        assert bits_equal(s.field(), before)
        s.step(4)
        got = s.field()
    with H.Solver(kappa, u0, h, dt, precision=prec) as ref:
        ref.step(8)
        assert bits_equal(got, ref.field())
