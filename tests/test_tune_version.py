"""A tuning cache says which kernels it timed; choices made for others are not taken."""
from __future__ import annotations

import json

import pytest

ENTRY = ' {"form": 3, "nz_max": 128, "kchunk": 24, "rows": 2, "minb": 3, "depth": 2, "glups": 1.0}'
TUNED = {"kchunk": 24, "rows": 2, "blocks_per_sm": 3, "depth": 2}
DEFAULT = {"kchunk": 32, "rows": 1, "blocks_per_sm": 4, "depth": 1}


@pytest.mark.parametrize("head,expected", [('{"device": "x", "entries": [', TUNED),
                                           ('{"device": "x", "kernels": 1, "entries": [', DEFAULT),
                                           ('{"device": "x", "kernels": 2, "entries": [', TUNED),
                                           ('{"device": "x", "kernels": 3, "entries": [', DEFAULT)])
def test_versions(heat, tmp_path, monkeypatch, head, expected):
    cache = tmp_path / "t.json"
    cache.write_text(f"{head}\n{ENTRY}\n]}}\n")
    monkeypatch.setenv("HEAT_TUNE_CACHE", str(cache))
    assert heat.tune_choice(heat.HEAT_FP32C, 0, 100) == expected


@pytest.mark.gpu
def test_a_written_cache_is_read_again(heat, cuda_device, tmp_path, monkeypatch):
    cache = tmp_path / "t.json"
    monkeypatch.setenv("HEAT_TUNE_CACHE", str(cache))
    heat.tune_batch(heat.HEAT_FP64, 0, max_nz=64, force=True)
    doc = json.loads(cache.read_text())
    entry = doc["entries"][0]
    assert doc["kernels"] == 2 and entry["kchunk"] <= 32 and entry["rows"] == 1
    again = tmp_path / "again.json"
    again.write_text(cache.read_text())
    monkeypatch.setenv("HEAT_TUNE_CACHE", str(again))
    assert heat.tune_choice(heat.HEAT_FP64, 0, 64)["kchunk"] == entry["kchunk"]
