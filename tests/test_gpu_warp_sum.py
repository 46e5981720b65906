"""The QR's integer warp sum against exact sums.

A term is rounded to the nearest multiple of 2^(E - 56), 2^E <= max |v|: 31
terms below the largest, half a unit each, and the sum's own rounding and that
of the reference's, so the two differ by at most 31 2^(E - 57) + 2^-52 |sum|.
The error is no more than the worst case of a tree of five FP64 additions,
5 2^-53 sum |v|, and its mean square stays under the tree's."""
import ctypes
import math
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "warp_sum.cuh"
__global__ void k(const double* in, double* out) {
  const int i = blockIdx.x * 32 + threadIdx.x;
  out[i] = pqmc::warp_sum(in[i]);
}
extern "C" int sums(int n, const double* in, double* out) {
  double *a = nullptr, *b = nullptr;
  const size_t bytes = sizeof(double) * 32 * (size_t)n;
  if (cudaMalloc(&a, bytes) || cudaMalloc(&b, bytes) || cudaMemcpy(a, in, bytes, cudaMemcpyHostToDevice)) return 1;
  k<<<n, 32>>>(a, b);
  const int st = cudaMemcpy(out, b, bytes, cudaMemcpyDeviceToHost);
  cudaFree(a);
  cudaFree(b);
  return st;
}
"""


@pytest.fixture(scope="module")
def sums(tmp_path_factory):
    from pqmc_allinone_gb300 import build as b
    d = tmp_path_factory.mktemp("warp_sum")
    (d / "s.cu").write_text(SOURCE)
    subprocess.run([b.nvcc(), *b.ARCH, *b.FLAGS, "-I", b.CSRC, "-shared", str(d / "s.cu"), "-o", str(d / "s.so"), "-lcudart"],
                   check=True, timeout=300)
    fn = ctypes.CDLL(str(d / "s.so")).sums
    fn.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]

    def call(v):
        v = np.ascontiguousarray(v, dtype=np.float64)
        out = np.empty_like(v)
        assert fn(len(v), v.ctypes.data, out.ctypes.data) == 0
        assert np.array_equal(out, np.repeat(out[:, :1], 32, axis=1), equal_nan=True)   # every lane has it
        return out[:, 0]
    return call


def _tree(v):
    v = v.copy()
    while v.shape[1] > 1:
        v = v[:, :v.shape[1] // 2] + v[:, v.shape[1] // 2:]
    return v[:, 0]


@pytest.mark.parametrize("scale", [-960, -500, 0, 500, 1000])
@pytest.mark.parametrize("spread", [0, 5, 30, 100])
def test_error_bound(sums, scale, spread):
    rng = np.random.default_rng(1000 * spread + scale + 5000)
    n = 4000
    spread = min(spread, 1000 + scale)   # magnitudes stay above 2^-1022
    v = np.ldexp(rng.normal(size=(n, 32)), scale - rng.integers(0, spread + 1, size=(n, 32)))
    v[: n // 4, 16:] = -v[: n // 4, :16] * (1 + np.ldexp(rng.normal(size=(n // 4, 16)), -40))   # cancelling
    got, exact = sums(v), np.array([math.fsum(r) for r in v])
    e = np.floor(np.log2(np.abs(v).max(axis=1)))
    # what falls below 2^-1022 is flushed
    bound = 31 * np.ldexp(1.0, (e - 57).astype(int)) + 2.0**-52 * np.abs(exact) + 2.0**-1022
    assert np.all(np.abs(got - exact) <= bound)
    total = np.abs(v).sum(axis=1)
    assert np.sqrt(np.mean(((got - exact) / total)**2)) <= np.sqrt(np.mean(((_tree(v) - exact) / total)**2))


def test_special_values(sums):
    v = np.zeros((8, 32))
    v[1, 3] = np.nan
    v[2, 7] = np.inf
    v[3, 0], v[3, 1] = np.inf, -np.inf
    v[4, :] = 1.7e308                 # past the range
    v[5, 5] = -5e-324                 # below 2^-1022: 0
    v[6, 2], v[6, 9] = 3.0, -3.0
    v[7, :] = -0.5
    s = sums(v)
    assert s[0] == 0.0 and np.isnan(s[1]) and np.isnan(s[2]) and np.isnan(s[3])
    assert s[4] == np.inf and s[5] == 0.0 and s[6] == 0.0 and s[7] == -16.0
