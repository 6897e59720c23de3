"""The bilinear sum of a texture lookup (texture_albedo, shading.cuh) keeps its
products unrounded. A texture of one column and two rows whose first texel is
-1, looked up at v = 1 - k / 1024: both weights and the first product are exact
in float, so the fused sum is the exact value rounded once, however far its two
products cancel, and the comparison is for equality."""
import subprocess

import numpy as np
import pytest

from renderer_gb300.build import ARCH, COMMON, CSRC, FLAGS, nvcc

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "shading.cuh"
__global__ void k(gbrt::DeviceScene S, gbrt::DevMaterial m, const float* v, int n, float* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  m.tex = i;
  const gbrt::V3f r = gbrt::texture_albedo(S, m, 0.f, v[i]);
  out[3 * i] = r.x;
  out[3 * i + 1] = r.y;
  out[3 * i + 2] = r.z;
}
int main() {
  int n;
  if (std::scanf("%d", &n) != 1 || n <= 0) return 1;
  std::vector<float> v(n), tex(6 * n), out(3 * n);
  std::vector<int4> info(n);
  for (int i = 0; i < n; ++i) {
    if (std::scanf("%f", &v[i]) != 1) return 1;
    for (int c = 0; c < 3; ++c) {
      tex[6 * i + c] = -1.f;
      if (std::scanf("%f", &tex[6 * i + 3 + c]) != 1) return 1;
    }
    info[i] = make_int4(2 * i, 1, 2, 0);
  }
  float *dv, *dt, *dout;
  int4* di;
  if (cudaMalloc(&dv, n * 4) || cudaMalloc(&dt, 6 * n * 4) || cudaMalloc(&dout, 3 * n * 4) || cudaMalloc(&di, n * 16))
    return 2;
  cudaMemcpy(dv, v.data(), n * 4, cudaMemcpyHostToDevice);
  cudaMemcpy(dt, tex.data(), 6 * n * 4, cudaMemcpyHostToDevice);
  cudaMemcpy(di, info.data(), n * 16, cudaMemcpyHostToDevice);
  gbrt::DeviceScene S{};
  S.tex_texels = dt;
  S.tex_info = di;
  gbrt::DevMaterial m{};
  m.kd[0] = m.kd[1] = m.kd[2] = 1.f;
  m.exponent = 1.f;
  k<<<(n + 127) / 128, 128>>>(S, m, dv, n, dout);
  if (cudaMemcpy(out.data(), dout, 3 * n * 4, cudaMemcpyDeviceToHost)) return 3;
  for (float x : out) std::printf("%.9g\n", x);
}
"""


def test_sum_is_rounded_once(tmp_path):
    (tmp_path / "p.cu").write_text(PROGRAM)
    subprocess.run([nvcc(), *ARCH, *COMMON, *FLAGS["pathtrace.cu"], "-I", CSRC, str(tmp_path / "p.cu"), "-o",
                    str(tmp_path / "p")], check=True, capture_output=True)
    rng = np.random.default_rng(7)
    n = 2000
    b = rng.integers(1, 1024, n) / 1024.0
    # second texels near the one that cancels the first, and far from it
    t = (1 - b)[:, None] / b[:, None] * (1 + rng.choice([1e-5, 1e-3, 0.3], (n, 3)) * rng.normal(size=(n, 3)))
    t = t.astype(np.float32)
    text = "%d\n" % n + "\n".join("%.9g %.9g %.9g %.9g" % (1 - x, *y) for x, y in zip(b, t))
    r = subprocess.run([str(tmp_path / "p")], input=text, capture_output=True, text=True)
    assert r.returncode == 0, r.returncode
    got = np.array(r.stdout.split(), np.float32).reshape(n, 3)
    want = (t.astype(np.float64) * b[:, None] - (1 - b)[:, None]).astype(np.float32)  # exact before its one rounding
    np.testing.assert_array_equal(got, want)
