"""What bench.py reports beside the headline figure of the default FP64 form: its
FP64-pipe work, seven conversions for four points, and the DRAM traffic that a profile
recorded."""
from __future__ import annotations

import importlib.util

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench", ROOT / "bench.py")
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    return module


def test_fp64_pipe_work_of_the_fixed_point_form(bench):
    r = bench.fx_pipe_record(10, 1.0, 100.0)
    assert r["ops_per_launch"] == 8 ** 3 * 7 / 4
    r = bench.fx_pipe_record(512, 0.8, 500.0)
    assert r["achieved_gops"] == pytest.approx(510 ** 3 * 7 / 4 / 0.8e-3 / 1e9, abs=0.1)
    assert r["frac"] == pytest.approx(r["achieved_gops"] / 500.0, rel=1e-3)
    assert bench.fx_pipe_record(10, 1.0, 0.0)["frac"] is None


def test_traffic_record_of_the_fixed_point_form(bench):
    # at least the field, its weights and the result once each, at most the halos on top
    t, source = bench.profile_traffic(510 ** 3, bench.FX_TRAFFIC_RECORD)
    assert 24 <= source["bytes_per_update"] <= 36
    assert t == pytest.approx(source["bytes_per_update"] * 510 ** 3, rel=1e-3)
