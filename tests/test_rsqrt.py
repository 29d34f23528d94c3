"""The FP64 reciprocal square root of the pair kernels, alone, against extended precision."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from beastgpu_gb300.csrc import build

SOURCE = r"""
#include "bgb_common.cuh"
__global__ void k(const double* x, double* y, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = bgb::rsqrt_newton(x[i]);
}
extern "C" int run(const double* x, double* y, int n) {
  double *dx = nullptr, *dy = nullptr;
  int rc = cudaMalloc(&dx, 8 * (size_t)n) || cudaMalloc(&dy, 8 * (size_t)n);
  rc = rc || cudaMemcpy(dx, x, 8 * (size_t)n, cudaMemcpyHostToDevice);
  if (!rc) k<<<(n + 255) / 256, 256>>>(dx, dy, n);
  rc = rc || cudaGetLastError() || cudaMemcpy(y, dy, 8 * (size_t)n, cudaMemcpyDeviceToHost);
  cudaFree(dx);
  cudaFree(dy);
  return rc;
}
"""


@pytest.mark.gpu
def test_rsqrt_newton(tmp_path):
    src, so = tmp_path / "r.cu", tmp_path / "r.so"
    src.write_text(SOURCE)
    subprocess.check_call([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, "-I", os.path.dirname(build.__file__), "-shared",
                           "-o", str(so), str(src)])
    rng = np.random.default_rng(1)
    x = np.ldexp(rng.uniform(1.0, 2.0, 400_000), rng.integers(-1021, 1023, 400_000))
    edges = np.ldexp(1.0, np.arange(-1022, 1024))
    x = np.concatenate([x, rng.uniform(0.25, 4.0, 400_000), edges, np.nextafter(edges[1:], 0.0), np.nextafter(edges, np.inf)])
    y = np.empty_like(x)
    assert ctypes.CDLL(str(so)).run(ctypes.c_void_p(x.ctypes.data), ctypes.c_void_p(y.ctypes.data), x.size) == 0
    exact = 1 / np.sqrt(x.astype(np.longdouble))
    # the last rounding (2^-53 of the result at most), the dropped term, and roundings of the correction far below it
    assert np.abs(y / exact - 1).max() <= 2.0 ** -53 + 2.0 ** -58
