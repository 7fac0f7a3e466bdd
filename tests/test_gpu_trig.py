"""The table-driven exponential and sine-cosine pair of the float64 Green function against 64-bit
mantissas, beside CUDA's functions on the same arguments."""
import os
import subprocess

import numpy as np
import pytest

from fourierd3_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cstdio>
#include <vector>
#include "fd3_common.cuh"
using namespace fd3;
__global__ void evaluate(int n, const Tables* tab, const double* x, const double* a, double* o) {
  __shared__ __align__(16) double t[TabTrig::kDoubles];
  TabTrig::fill(t, tab);
  __syncthreads();
  const TabTrig tr{t};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    o[i] = tr.expv(x[i]);
    tr.sincospiv(a[i], o + n + i, o + 2 * n + i);
    o[3 * n + i] = exp(x[i]);
    sincospi(a[i], o + 4 * n + i, o + 5 * n + i);
  }
}
int main(int argc, char** argv) {
  const int n = atoi(argv[1]);
  std::vector<double> h(6 * (size_t)n);
  FILE* f = fopen(argv[2], "rb");
  if (fread(h.data(), 16, n, f) != (size_t)n) return 1;
  fclose(f);
  double *in, *out;
  Tables* tab;
  static Tables ht;
  TabTrig::make(ht.trig);
  if (cudaMalloc(&in, 16 * (size_t)n) || cudaMalloc(&out, 48 * (size_t)n) || cudaMalloc(&tab, sizeof(ht))) return 1;
  cudaMemcpy(in, h.data(), 16 * (size_t)n, cudaMemcpyHostToDevice);
  cudaMemcpy(tab, &ht, sizeof(ht), cudaMemcpyHostToDevice);
  evaluate<<<148, 256>>>(n, tab, in, in + n, out);
  if (cudaMemcpy(h.data(), out, 48 * (size_t)n, cudaMemcpyDeviceToHost)) return 1;
  f = fopen(argv[3], "wb");
  return fwrite(h.data(), 48, n, f) == (size_t)n && fclose(f) == 0 ? 0 : 1;
}
"""


def test_tables_are_no_further_off_than_the_library_functions(cuda_device, tmp_path):
    src, exe = tmp_path / "trig.cu", tmp_path / "trig"
    src.write_text(SOURCE)
    subprocess.run([build.NVCC, "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "--expt-relaxed-constexpr", "-I" + build.CSRC, str(src), "-o", str(exe)], check=True)
    n, rng = 600000, np.random.default_rng(0)
    # u = k R up to 600: the exponentials' arguments, the phases in half turns, and the ends of the table's arcs
    x = -rng.random(n) * np.repeat([1.0, 20.0, 600.0], n // 3)
    a = 0.25 + rng.random(n) * np.repeat([1.0, 20.0, 300.0], n // 3)
    x[:65], a[:129] = -np.log(2.0) * np.arange(65) / 64, (np.arange(129) + 0.5) / 32
    np.concatenate((x, a)).tofile(tmp_path / "in")
    subprocess.run([str(exe), str(n), str(tmp_path / "in"), str(tmp_path / "out")], check=True, env=dict(os.environ))
    out = np.fromfile(tmp_path / "out").reshape(2, 3, n)
    pi = np.longdouble("3.14159265358979323846264338327950288")
    ex, phase = np.exp(np.longdouble(x)), pi * np.longdouble(np.fmod(a, 2.0))
    want = np.stack((ex, np.sin(phase), np.cos(phase)))
    err = np.abs(out - want)
    err[:, 0] /= ex
    for ours, cuda in ((err[0, 0], err[1, 0]), (err[0, 1:], err[1, 1:])):
        assert ours.max() <= cuda.max() and (ours**2).mean() <= (cuda**2).mean()
    # one rounding to double, and a twentieth of one for what comes before it (sines: |v| <= 1, 2^-54, and the
    # rounding of the rotation by up to pi / 64)
    assert err[0, 0].max() <= 1.05 * 2.0**-53 and err[0, 1:].max() <= 1.5 * 2.0**-54
