"""Grids of very many planes: no launch asks for more z-chunks than a CUDA grid may
have (65,535), whatever the chunk rule would like best."""
from __future__ import annotations

import subprocess

import numpy as np
import pytest

from conftest import PKG, ROOT, bits_equal

PROGRAM = r"""
#include <cstdio>
#include "heat_internal.h"
int main() {
  int bad = 0;
  const int most[] = {10, 32, 128};          // bit-exact, fixed point, two-step FP32C
  const int interior[] = {1, 2, 31, 510, 65535, 65536, 655349, 655351, 699998, 2097119, 2097121,
                          8388481, 20000000, 715827880};
  for (int m : most)
    for (int n : interior)
      for (long tiles : {1L, 7L, 4096L, 1000000L})
        for (long resident : {0L, 152L, 608L, 1824L}) {
          const int kc = heat::balanced_chunk(tiles, n, resident, 1, 0.5, m);
          const bool fits = kc >= 1 && (n + kc - 1) / kc <= 65535;
          const bool short_ok = n > 65535 * m || kc <= m || resident == 0;
          if (!fits || !short_ok) ++bad, std::printf("%d planes, most %d: %d\n", n, m, kc);
        }
  return bad != 0;
}
"""


def test_chunk_rule(tmp_path):
    import heat_build
    src, exe = tmp_path / "chunks.cpp", tmp_path / "chunks"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(ROOT / "include"), "-I", str(PKG / "csrc"), "-I",
                    str(heat_build._cuda_include(heat_build._nvcc())), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[:2000]


STEPS = 3


@pytest.mark.gpu
@pytest.mark.parametrize("planes", [655_353, 700_000])
def test_bitexact_forms(heat, oracle, cuda_device, planes):
    torch, H = cuda_device, heat
    kappa, u0, h, dt = H.inputs_config(0, 5, 3, 3, planes)
    ref = oracle.steps(u0, kappa, h, dt, STEPS)
    with H.Solver(kappa, u0, h, dt, flags=H.HEAT_BITEXACT) as s:
        s.step(STEPS)
        assert bits_equal(s.field(), ref)
    a, k = torch.from_numpy(u0).cuda(), torch.from_numpy(kappa).cuda()
    b = a.clone()
    for _ in range(STEPS):
        H.check(H.lib().heat_update(b.data_ptr(), a.data_ptr(), None, k.data_ptr(), planes, 3, 3,
                                    oracle.factor(h, dt), 0), "heat_update")
        a, b = b, a
    torch.cuda.synchronize()
    assert bits_equal(a.cpu().numpy(), ref)


@pytest.mark.gpu
@pytest.mark.parametrize("planes", [2_097_123, 2_200_000])
def test_default_form(heat, oracle, cuda_device, planes):
    H = heat
    kappa, u0, h, dt = H.inputs_config(0, 6, 3, 3, planes)
    ref = oracle.steps(u0, kappa, h, dt, STEPS)
    with H.Solver(kappa, u0, h, dt) as s:
        s.step(STEPS)
        got = s.field()
    # a rounding and about one unit of the last place a step, the oracle's seven
    assert np.abs(got - ref).max() <= STEPS * 5 * 2.0 ** -52 * np.abs(u0).max()


@pytest.mark.gpu
def test_default_form_in_tiles(heat, oracle, cuda_device):
    """Three rows: the tiled kernel, in two launches a step."""
    H = heat
    kappa, u0, h, dt = H.inputs_config(0, 7, 3, 5, 2_100_000)
    ref = oracle.steps(u0, kappa, h, dt, STEPS)
    with H.Solver(kappa, u0, h, dt) as s:
        s.step(STEPS)
        got = s.field()
        assert H.lib().heat_diag_fp64_timeout(s._ctx) == H.HEAT_OK  # it steps with that kernel
        assert H.lib().heat_sync(s._ctx) == H.HEAT_ETIMEOUT
    assert np.abs(got - ref).max() <= STEPS * 5 * 2.0 ** -52 * np.abs(u0).max()
