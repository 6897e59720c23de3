"""The texel index of an environment lookup (env_texel, shading.cuh) for maps
of more than 2^31 texels, which gbrt_scene_create accepts: the function runs on
the host here, no map is allocated.

The directions look at texel centres far from any edge of a texel, so float
rounding cannot change the texel."""
import subprocess

import numpy as np
import pytest

from renderer_gb300 import _abi
from renderer_gb300.build import ARCH, COMMON, CSRC, nvcc

PROGRAM = r"""
#include <cstdio>
#include "shading.cuh"
int main() {
  int w, h, mapping;
  float x, y, z;
  while (std::scanf("%d %d %d %f %f %f", &w, &h, &mapping, &x, &y, &z) == 6)
    std::printf("%lld\n", (long long)gbrt::env_texel(w, h, mapping, x, y, z));
}
"""


@pytest.fixture(scope="module")
def env_texel(tmp_path_factory):
    d = tmp_path_factory.mktemp("env_texel")
    (d / "p.cu").write_text(PROGRAM)
    subprocess.run([nvcc(), *ARCH, *COMMON, "-I", CSRC, str(d / "p.cu"), "-o", str(d / "p")], check=True,
                   capture_output=True)

    def run(cases):
        text = "\n".join(" ".join(repr(v) for v in c) for c in cases)
        r = subprocess.run([str(d / "p")], input=text, capture_output=True, text=True, check=True)
        return [int(v) for v in r.stdout.split()]
    return run


@pytest.mark.parametrize("w,h", [(64, 32), (46340, 46341), (46341, 46341), (70000, 40000), (100001, 65521)])
def test_latlong(env_texel, w, h):
    rng = np.random.default_rng(w)
    cases, want = [], []
    for _ in range(20):
        # a cell of a coarse grid, whose centre's texel is known up to the
        # rounding of the angles: compare the row and the column to 1e-5
        u, v = rng.uniform(0.05, 0.95, 2)
        th, ph = np.pi * v, 2 * np.pi * (u - 0.5)
        cases.append((w, h, _abi.ENV_LATLONG, float(np.sin(th) * np.sin(ph)), float(np.cos(th)),
                      float(-np.sin(th) * np.cos(ph))))
        want.append((v * h, u * w))
    for i, (row, col) in zip(env_texel(cases), want):
        assert 0 <= i < w * h
        assert abs(i // w + 0.5 - row) < 0.5 + 1e-5 * h and abs(i % w + 0.5 - col) < 0.5 + 1e-5 * w


@pytest.mark.parametrize("n", [64, 46341, 65521, 100001])
def test_angular(env_texel, n):
    # The probe's centre is +x; a direction theta off it towards y lies
    # theta / pi of the half side from the centre.
    cases, want = [], []
    for th in np.linspace(0.1, 3.0, 13):
        for a in (0.4, 2.0, 4.4):
            y, z = np.sin(th) * np.cos(a), -np.sin(th) * np.sin(a)
            cases.append((n, n, _abi.ENV_ANGULAR, float(np.cos(th)), float(y), float(z)))
            cx, cy = th / np.pi * np.cos(a), th / np.pi * np.sin(a)
            want.append(((cy + 1) / 2 * n - 1, (cx + 1) / 2 * n - 1))
    for i, (row, col) in zip(env_texel(cases), want):
        assert 0 <= i < n * n
        assert abs(i // n + 0.5 - row) < 0.5 + 1e-5 * n and abs(i % n + 0.5 - col) < 0.5 + 1e-5 * n
