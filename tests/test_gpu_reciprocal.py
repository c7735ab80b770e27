"""The Poisson multiplier's reciprocal equals CUDA's correctly rounded one, and
the float64 quotient rounded to float32, for every float of the range that the
wavenumber tables keep to: 2^23 mantissas, exponents 0 to 28."""
import ctypes
import subprocess

import pytest

from ns_solver_jax_differential_distributed_gb300 import _build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "nsgb_fft_bodies.cuh"
__global__ void sweep(unsigned first, unsigned count, unsigned long long* bad) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const float d = __uint_as_float(first + i), r = nsgb::reciprocal(d);
    if (r != __frcp_rn(d)) atomicAdd(bad, 1ull);
    if (r != (float)(1.0 / (double)d)) atomicAdd(bad + 1, 1ull);
  }
}
extern "C" int count_bad(unsigned first, unsigned count, unsigned long long* out) {
  unsigned long long* d = nullptr;
  cudaError_t e = cudaMalloc(&d, 16);
  if (e == cudaSuccess) e = cudaMemset(d, 0, 16);
  if (e == cudaSuccess) sweep<<<1216, 256>>>(first, count, d);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpy(out, d, 16, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
"""


def test_reciprocal_is_correctly_rounded(cuda_lib, tmp_path):
    src, lib = tmp_path / "sweep.cu", tmp_path / "sweep.so"
    src.write_text(SOURCE)
    subprocess.run([_build.nvcc(), *_build.ARCH, *_build.NVFLAGS, "-shared", "-o", str(lib), str(src), "-lcudart"],
                   check=True, capture_output=True)
    fn = ctypes.CDLL(str(lib)).count_bad
    fn.argtypes = [ctypes.c_uint, ctypes.c_uint, ctypes.c_void_p]
    bad = (ctypes.c_ulonglong * 2)()
    for e in range(29):
        assert fn((127 + e) << 23, 1 << 23, bad) == 0
        assert (bad[0], bad[1]) == (0, 0), (e, bad[0], bad[1])
