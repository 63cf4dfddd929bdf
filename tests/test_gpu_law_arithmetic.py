"""dist_of and inv_sq (epi_b200/csrc/epi_common.cuh), which stand for the square
root and the division of the FP64 laws, against CUDA's correctly rounded ones.
A Newton step on an exact residual squares the error of its start (a reciprocal
square root good to an ulp or two, so 2^-51 becomes 2^-101) and rounds once:
within half an ulp and a little, so never more than one from the correctly
rounded value. Squared distances: all of the laws' range (contacts of a
hundredth of a radius to connections of 4), and far beyond it on either side."""
import ctypes
import subprocess

import numpy as np
import pytest

from epi_b200 import build as B

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "epi_common.cuh"
namespace epi {
__device__ __forceinline__ long long apart(double a, double b) {  // in ulps, same sign
  const long long d = __double_as_longlong(a) - __double_as_longlong(b);
  return d < 0 ? -d : d;
}
__global__ void k(const double* d2, int n, long long* most) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double inv = lrsqrt(d2[i]);
    atomicMax(most, apart(dist_of(d2[i], inv), __dsqrt_rn(d2[i])));
    atomicMax(most + 1, apart(inv_sq(d2[i], inv), __ddiv_rn(1.0, d2[i])));
  }
}
}  // namespace epi
extern "C" int run(const double* h, int n, long long* most) {
  double* d;
  long long* m;
  cudaMalloc(&d, sizeof(double) * n);
  cudaMalloc(&m, 2 * sizeof(long long));
  cudaMemcpy(d, h, sizeof(double) * n, cudaMemcpyHostToDevice);
  cudaMemset(m, 0, 2 * sizeof(long long));
  epi::k<<<256, 256>>>(d, n, m);
  cudaMemcpy(most, m, 2 * sizeof(long long), cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(m);
  return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("laws")
    (d / "laws.cu").write_text(SOURCE)
    subprocess.run([B.nvcc(), *B.ARCH, "-O3", "-std=c++17", "--shared", "-Xcompiler", "-fPIC",
                    "-I", str(B.CSRC), "-o", str(d / "laws.so"), str(d / "laws.cu")], check=True)
    return ctypes.CDLL(str(d / "laws.so")).run


@pytest.mark.parametrize("low,high", [(1e-4, 16.0), (1e-300, 1e300)])
def test_within_an_ulp_of_square_root_and_division(run, low, high):
    rng = np.random.default_rng(7)
    d2 = np.exp(rng.uniform(np.log(low), np.log(high), 4_000_000))
    most = (ctypes.c_longlong * 2)()
    assert run(d2.ctypes.data_as(ctypes.c_void_p), d2.size, most) == 0
    assert most[0] <= 1 and most[1] <= 1, list(most)


def test_zero_and_the_smallest_distances(run):
    """0 and infinity as a square root and a division give them; below 2^-1022
    / 4 the inverse overflows in both."""
    d2 = np.array([0.0, 5e-324, 1e-320, 1e-309])
    most = (ctypes.c_longlong * 2)()
    assert run(d2.ctypes.data_as(ctypes.c_void_p), d2.size, most) == 0
    assert most[1] == 0
    assert run(d2.ctypes.data_as(ctypes.c_void_p), 1, most) == 0
    assert most[0] == 0 and most[1] == 0
