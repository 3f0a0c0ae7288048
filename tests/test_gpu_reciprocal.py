"""The eliminations' pivot reciprocal (csrc/common.cuh: crecip) against 1 / d in extended
precision over the exponents of a double.  Bound of each part: |s d|^2 is off by 2 units of
2^-53 (one product, one multiply-add), its reciprocal after the last Newton step by 2 (the
residual's and the step's rounding), the product by 1: 5, and 6 with the second order."""
from __future__ import annotations

import ctypes
import subprocess
import textwrap

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SOURCE = textwrap.dedent("""
    #include <cuda_runtime.h>
    #include "common.cuh"
    static __global__ void k(const trhepd::cd* d, trhepd::cd* r, int n) {
      const int i = blockIdx.x * blockDim.x + threadIdx.x;
      if (i < n) r[i] = trhepd::crecip(d[i]);
    }
    extern "C" int reciprocals(const void* d, void* r, int n) {
      void *a = nullptr, *b = nullptr;
      const size_t bytes = (size_t)n * sizeof(trhepd::cd);
      cudaMalloc(&a, bytes);
      cudaMalloc(&b, bytes);
      cudaMemcpy(a, d, bytes, cudaMemcpyHostToDevice);
      k<<<(n + 127) / 128, 128>>>((const trhepd::cd*)a, (trhepd::cd*)b, n);
      cudaMemcpy(r, b, bytes, cudaMemcpyDeviceToHost);
      cudaFree(a);
      cudaFree(b);
      return (int)cudaGetLastError();
    }
""")


def test_reciprocal(tmp_path):
    from trhepd_opt_b200 import build
    (tmp_path / "r.cu").write_text(SOURCE)
    lib = tmp_path / "libr.so"
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-I", str(build.CSRC), str(tmp_path / "r.cu"), "-o", str(lib)],
                   check=True)
    rng = np.random.default_rng(1)
    n = 200001
    # parts of like size, of very unlike sizes, and one of them zero
    e = rng.integers(-1020, 1000, n)
    gap = np.where(rng.random(n) < 0.5, 0, rng.integers(-60, 1, n))
    d = np.ldexp(rng.uniform(1, 2, n), e) * rng.choice([-1, 1], n) + 1j * np.ldexp(
        rng.uniform(1, 2, n), np.maximum(e + gap, -1022)) * rng.choice([-1, 1], n)
    d[::7] = d[::7].real
    d[1::7] = 1j * d[1::7].imag
    r = np.zeros_like(d)
    f = ctypes.CDLL(str(lib)).reciprocals
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int]
    assert f(d.ctypes.data, r.ctypes.data, n) == 0
    # 64-bit mantissa, 15-bit exponent: the squares neither overflow nor underflow
    x, y = d.real.astype(np.longdouble), d.imag.astype(np.longdouble)
    q = x * x + y * y
    for got, ref in ((r.real, x / q), (r.imag, -y / q)):
        normal = np.abs(ref) > 2.0 ** -1021  # smaller parts round to subnormals
        off = np.abs(got.astype(np.longdouble) - ref)[normal] / np.abs(ref[normal])
        assert off.max() <= 6 * 2.0 ** -53, float(off.max())
        assert np.all(np.abs(got[~normal] - ref[~normal].astype(float)) <= 2.0 ** -1073)
