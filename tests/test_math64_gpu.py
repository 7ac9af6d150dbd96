"""csrc/math64.cuh and csrc/cvt.cuh on the GPU: the FP64 exponential and quotient of the HH
rates, and the integer FP32 <-> FP64 conversions.

A small program compiled here with nvcc evaluates them over arrays from the host.  exp64 is held
to 0.6 ulp of the exponential in extended precision (its derivation: half an ulp of rounding
plus 0.06 of the table's and the FP32 bracket's share) and div64 to the correctly rounded
quotient; the conversions give numpy's result bit for bit.  Arguments off the short paths
(overflow, zero, infinities, NaN, subnormals) are among them."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SRC = r"""
#include <cstdio>
#include <vector>
#include "math64.cuh"
__global__ void eval(int n, const double *a, const double *b, double *o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  o[i] = nrt::exp64(a[i]);
  o[n + i] = nrt::div64(a[i], b[i]);
  o[2 * n + i] = nrt::f2d(nrt::d2f(b[i]));
  o[3 * n + i] = nrt::exp64(a[i], -3);
}
int main(int, char **v) {
  FILE *f = fopen(v[1], "rb");
  int n;
  if (fread(&n, 4, 1, f) != 1) return 1;
  std::vector<double> h(2 * n), o(4 * n);
  if (fread(h.data(), 8, 2 * n, f) != (size_t)(2 * n)) return 1;
  fclose(f);
  double *d, *e;
  cudaMalloc(&d, 16 * n);
  cudaMalloc(&e, 32 * n);
  cudaMemcpy(d, h.data(), 16 * n, cudaMemcpyHostToDevice);
  eval<<<(n + 255) / 256, 256>>>(n, d, d + n, e);
  if (cudaMemcpy(o.data(), e, 32 * n, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  f = fopen(v[2], "wb");
  fwrite(o.data(), 8, 4 * n, f);
  fclose(f);
  return 0;
}
"""


def test_exp_quotient_and_conversions(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cu, exe = tmp_path / "m.cu", tmp_path / "m"
    cu.write_text(SRC)
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I",
                    os.path.join(ROOT, "168861_gb300", "csrc"), "-o", str(exe), str(cu)], check=True)
    rng = np.random.default_rng(3)
    special = np.array([0.0, -0.0, 1e-300, 5e-324, np.inf, -np.inf, np.nan, 709.9, 690.5, -745.2,
                        1e-40, -1.5e-45, 7e-46, 3.5e38, 1e300, 2.0 ** -126, 2.0 ** 128])
    a = np.concatenate([rng.uniform(-25, 25, 200000), rng.uniform(-1e-3, 1e-3, 100000),
                        rng.uniform(-700, 700, 100000), special, rng.permutation(special)])
    b = np.concatenate([np.expm1(rng.uniform(-20, 20, 400000)) * rng.choice([1, 1e-30, 1e20], 400000),
                        rng.permutation(special), special])
    (tmp_path / "in").write_bytes(np.int32(len(a)).tobytes() + a.tobytes() + b.tobytes())
    subprocess.run([str(exe), str(tmp_path / "in"), str(tmp_path / "out")], check=True)
    e, q, c, e3 = np.fromfile(tmp_path / "out").reshape(4, -1)
    with np.errstate(all="ignore"):
        want = np.exp(a.astype(np.longdouble))
        w64 = np.exp(a)
        ok = np.isfinite(w64) & (w64 > 1e-300)
        ulp = np.abs(e[ok] - want[ok]) / np.spacing(w64[ok])
        assert ulp.max() < 0.6 if np.finfo(np.longdouble).nmant > 52 else 1.6
        np.testing.assert_array_equal(e[~ok & (w64 == 0)], 0.0)
        np.testing.assert_array_equal(np.isposinf(e), np.isposinf(w64))
        np.testing.assert_array_equal(np.isnan(e), np.isnan(a))
        np.testing.assert_array_equal(e3[ok], e[ok] / 8)
        np.testing.assert_array_equal(q, a / b)
        np.testing.assert_array_equal(c, b.astype(np.float32).astype(np.float64))
