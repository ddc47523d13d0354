"""rcp_nr and sqrt_nr, which every FP64 flux, density and conversion goes through, against
1/x and sqrt(x).

Both end with one fused rounding of a value whose relative error is below 2^-75, so a result is
the correctly rounded one or its neighbour: one unit in the last place is the bound, over random
mantissas with exponents from -900 to 900 of either sign, powers of two and their neighbours.
Zeros, infinities and NaN give NaN, as their comment says: a state that holds one is flagged.
"""
import ctypes as C
import subprocess

import numpy as np
import pytest

from tensum_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cuda_runtime.h>
#include "tg_physics.cuh"
__global__ void k(const double* x, double* r, double* s, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  r[i] = tg::rcp_nr(x[i]);
  s[i] = tg::sqrt_nr(fabs(x[i]));
}
extern "C" int evaluate(const double* x, double* r, double* s, int n) {
  double* d = nullptr;
  const size_t b = n * sizeof(double);
  cudaError_t e = cudaMalloc((void**)&d, 3 * b);
  if (e == cudaSuccess) e = cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k<<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * (size_t)n, n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(r, d + n, b, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(s, d + 2 * (size_t)n, b, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
"""


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    d = tmp_path_factory.mktemp("rcp")
    (d / "rcp.cu").write_text(SOURCE)
    so = d / "rcp.so"
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "--expt-relaxed-constexpr", "-I", build.CSRC, "-o", str(so), str(d / "rcp.cu")], check=True)
    f = C.CDLL(str(so)).evaluate
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int]

    def run(x):
        x = np.ascontiguousarray(x, np.float64)
        r, s = np.empty_like(x), np.empty_like(x)
        assert f(x.ctypes.data, r.ctypes.data, s.ctypes.data, x.size) == 0
        return r, s
    return run


def _ulps(a, b):
    """Distance in units in the last place of two arrays whose signs agree."""
    assert np.array_equal(np.signbit(a), np.signbit(b)) and np.all(np.isfinite(a))
    return np.abs(np.abs(a).view(np.int64) - np.abs(b).view(np.int64))


@pytest.mark.parametrize("lo,hi", [(-900, 900), (-60, 60), (0, 1)])
def test_within_one_unit_in_the_last_place(evaluate, lo, hi):
    rng = np.random.default_rng(hi)
    n = 1 << 22
    x = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n)) * rng.choice([-1.0, 1.0], n)
    two = np.ldexp(1.0, np.arange(lo, hi))
    x = np.concatenate([x, two, np.nextafter(two, 0.0), np.nextafter(two, np.inf)])
    r, s = evaluate(x)
    assert _ulps(r, 1.0 / x).max() <= 1
    assert _ulps(s, np.sqrt(np.abs(x))).max() <= 1


def test_outside_their_domain(evaluate):
    r, s = evaluate(np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324]))
    assert np.all(np.isnan(r)) and np.all(np.isnan(s))
