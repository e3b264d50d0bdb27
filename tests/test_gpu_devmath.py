"""Device arithmetic of devmath.cuh against 80-bit values and CUDA's rsqrt (needs a
B200: -m gpu): a small library with nothing but these functions is compiled.

Tolerances, from the operations of each: rsqrt_fast 1.5 2^-53 relative and its
series remainder (below 2^-58 for an approximation good to 2^-20); CUDA's rsqrt one
unit in the last place beside it.  cos x absolute, sin x relative: 4 and 5 times
2^-53 by half the angle (two factors of 2^-53 and the squares' or the product's
rounding), 2 and 3 for the series of x itself."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
U = 2.0 ** -53
SRC = r"""
#include "devmath.cuh"
__global__ void k(int n, const double *x, double *f, double *r, const double *t, double *cs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  f[i] = rsqrt_fast(x[i]);
  r[i] = rsqrt(x[i]);
  cossin_small(t[i], cs[4 * i], cs[4 * i + 1]);
  cossin_small_short(0.25 * t[i], cs[4 * i + 2], cs[4 * i + 3]);
}
extern "C" int run(int n, const double *x, double *f, double *r, const double *t, double *cs) {
  double *d;
  if (cudaMalloc(&d, 8 * sizeof(double) * (size_t)n) != cudaSuccess) return 1;
  cudaMemcpy(d, x, sizeof(double) * n, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, t, sizeof(double) * n, cudaMemcpyHostToDevice);
  k<<<(n + 127) / 128, 128>>>(n, d, d + 2 * n, d + 3 * n, d + n, d + 4 * n);
  cudaMemcpy(f, d + 2 * n, sizeof(double) * n, cudaMemcpyDeviceToHost);
  cudaMemcpy(r, d + 3 * n, sizeof(double) * n, cudaMemcpyDeviceToHost);
  cudaMemcpy(cs, d + 4 * n, 4 * sizeof(double) * n, cudaMemcpyDeviceToHost);
  const int e = (int)cudaGetLastError();
  cudaFree(d);
  return e;
}
"""


def test_device_functions(tmp_path):
    src, so = tmp_path / "m.cu", tmp_path / "m.so"
    src.write_text(SRC)
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-shared",
                    "-Xcompiler", "-fPIC", "-ccbin", "/usr/bin/g++", "-I", os.path.join(ROOT, "buff-em_b200", "csrc"),
                    "-o", str(so), str(src)], check=True)
    rng = np.random.default_rng(0)
    n = 1 << 20
    # mantissas of both octaves of the exponent's parity, neighbours of powers of two, the ends of the range
    x = np.ldexp(1 + rng.random(n), rng.integers(-1022, 1023, n))
    edge = np.ldexp(1.0, np.arange(-1020, 1023))
    x[:len(edge)], x[len(edge):2 * len(edge)], x[2 * len(edge):3 * len(edge)] = edge, np.nextafter(edge, 0), np.nextafter(edge, np.inf)
    x[-2:] = np.finfo(float).tiny, np.finfo(float).max
    t = np.r_[rng.uniform(-1, 1, n - 4), 1.0, -1.0, 1e-300, 0.0]
    f, r, cs = np.empty(n), np.empty(n), np.empty((n, 4))
    L = ctypes.CDLL(str(so))
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    assert L.run(n, p(x), p(f), p(r), p(t), p(cs)) == 0
    ref = 1 / np.sqrt(x.astype(np.longdouble))
    assert np.all(np.abs(f - ref) <= (1.5 + 0.03) * U * ref)
    assert np.all(np.abs(f - r) <= (1.5 + 0.03) * U * ref + np.spacing(r))
    for k, (a, c, s) in enumerate(((t, 4, 5), (0.25 * t, 2, 3))):
        a = a.astype(np.longdouble)
        assert np.all(np.abs(cs[:, 2 * k] - np.cos(a)) <= c * U)
        assert np.all(np.abs(cs[:, 2 * k + 1] - np.sin(a)) <= s * U * np.abs(np.sin(a)))
