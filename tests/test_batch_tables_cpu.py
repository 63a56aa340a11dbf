"""Uploads of the batch engine's tables, on a fake CUDA runtime (no GPU): a
copy may read its source at any time before something waits for it, so it must come
from page-locked memory that the batch owns and does not touch meanwhile."""
from __future__ import annotations

import os
import re
import subprocess

import pytest

from conftest import PKG, ROOT


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    import heat_build
    exe = tmp_path_factory.mktemp("batch") / "batch_tables"
    subprocess.run(["g++", "-g", "-O1", "-std=c++17", "-fsanitize=address", "-D_GLIBCXX_ASSERTIONS", "-I", str(ROOT / "include"),
                    "-I", str(PKG / "csrc"), "-I", str(heat_build._cuda_include(heat_build._nvcc())),
                    str(ROOT / "tests" / "batch_tables_fake.cpp"), str(PKG / "csrc" / "heat_batch_host.cpp"),
                    "-o", str(exe)], check=True)
    return exe


def test_table_uploads_read_memory_the_batch_keeps(program):
    env = {**os.environ, "ASAN_OPTIONS": "detect_leaks=0"}
    r = subprocess.run([str(program)], capture_output=True, text=True, env=env)
    assert r.returncode == 0, r.stdout + r.stderr


def test_tensor_maps_are_acquired_at_system_scope():
    """The table kernels' tensor maps are written by host copies into memory that held
    other maps before: an acquire at GPU scope does not order their use after that."""
    scopes = [(f.name, scope) for f in sorted((PKG / "csrc").iterdir()) if f.suffix in (".cu", ".cuh")
              for scope in re.findall(r"fence\.proxy\.tensormap::generic\.acquire\.(\w+)", f.read_text())]
    assert scopes and all(scope == "sys" for _, scope in scopes), scopes
