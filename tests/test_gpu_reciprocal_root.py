"""rcp_nr and sqrt_nr (csrc/common.cuh), which stand for the quotients and roots of the flux and limiter arithmetic:
their stated error over their stated range, and what they give outside it."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = """
#include "common.cuh"
__global__ void both(const double* x, double* r, double* s, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) { r[i] = mhd::rcp_nr(x[i]); s[i] = mhd::sqrt_nr(x[i]); }
}
extern "C" int evaluate(const double* x, double* r, double* s, int n) {
  double* d = nullptr;
  if (cudaMalloc(&d, 3 * sizeof(double) * n) != cudaSuccess) return 1;
  cudaMemcpy(d, x, sizeof(double) * n, cudaMemcpyHostToDevice);
  both<<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * n, n);
  cudaMemcpy(r, d + n, sizeof(double) * n, cudaMemcpyDeviceToHost);
  cudaMemcpy(s, d + 2 * n, sizeof(double) * n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return cudaGetLastError() != cudaSuccess;
}
"""


@pytest.fixture(scope="module")
def evaluate(pkg, tmp_path_factory):
    d = tmp_path_factory.mktemp("reciprocal_root")
    src, so = d / "both.cu", d / "both.so"
    src.write_text(SRC)
    csrc = os.path.join(os.path.dirname(pkg.__file__), "csrc")
    nvcc = "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else "nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-I", csrc, str(src), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    ptr = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731

    def run(x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        r, s = np.empty_like(x), np.empty_like(x)
        assert lib.evaluate(ptr(x), ptr(r), ptr(s), x.size) == 0
        return r, s
    return run


# against extended precision (11 bits more than the results have), relative.  Reciprocal: the final rounding,
# 2^-53, and the terms left out, below 0.02 of it; root: half of its first product's rounding more, and terms
# (5/2 t^3, t below 2^-20) of 0.02
UNIT = 2.0 ** -53


@pytest.mark.parametrize("kind", ["whole range", "one binade", "next to powers of two"])
def test_error_over_the_stated_range(evaluate, kind):
    rng = np.random.default_rng(7)
    n = 1 << 20
    if kind == "whole range":
        x = np.exp2(rng.uniform(-900.0, 900.0, n))
    elif kind == "one binade":
        x = np.concatenate([rng.uniform(1.0, 4.0, n), 1.0 + np.arange(4096) * 2.0 ** -52])
    else:
        k = np.arange(-900, 901).astype(float)
        x = np.concatenate([np.exp2(k) * (1.0 + m * 2.0 ** -52) for m in (-1, -0.5, 0, 1, 2)])
        x = x[(x >= 2.0 ** -900) & (x <= 2.0 ** 900)]
    r, s = evaluate(x)
    xl = x.astype(np.longdouble)
    assert np.finfo(np.longdouble).nmant >= 63
    assert np.abs(r.astype(np.longdouble) * xl - 1).max() <= 1.02 * UNIT
    root = np.sqrt(xl)
    assert (np.abs(s.astype(np.longdouble) - root) / root).max() <= 1.55 * UNIT
    assert np.array_equal(evaluate(-x)[0], -r)


def test_outside_the_range(evaluate):
    r, s = evaluate([0.0, -0.0, 5e-324, np.inf, -np.inf, np.nan])
    assert not np.isfinite(r).any() and not np.isfinite(s).any()
    assert np.isnan(evaluate([-1.0, -4.0])[1]).all()
    tiny = 1.0e-280  # what an argument that may be zero carries
    assert abs(evaluate([tiny])[1][0] - 1.0e-140) <= 4 * np.finfo(float).eps * 1.0e-140
