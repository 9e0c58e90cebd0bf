"""div_refined (csrc/fast_div.cuh) with divisors outside the range that the
flushing reciprocal covers: subnormal ones whose reciprocal is finite (2^-128 to
2^-126) and ones above 2^126, whose reciprocal is subnormal.  With a reciprocal
good to 2^-20 or better there the correction leaves an error of 2^-40 before the
last rounding, so the quotient is the IEEE one or its neighbour; numerators are
chosen so that quotient and residual stay clear of the subnormals."""
import ctypes as C
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "cudaprotoplanetarydisksfloat_b200", "csrc")

SRC = r'''
#include <cuda_runtime.h>
#include "fast_div.cuh"
// divisors first .. first + n - 1 by their bits, each with 64 numerators of exponent ex
__global__ void k_check(unsigned first, unsigned n, int ex, unsigned long long* bad) {
  for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const float y = __uint_as_float(first + k);
    for (unsigned m = 0; m < 64; m++) {
      const unsigned frac = (k * 2654435761u + m * 131071u * 40503u) & 0x7fffffu;
      const float x = __uint_as_float((unsigned)(ex + 127) << 23 | frac);
      const int a = (int)__float_as_uint(__fdiv_rn(x, y)), b = (int)__float_as_uint(div_refined(x, y));
      if (a - b > 1 || b - a > 1) atomicAdd(bad, 1ull);
    }
  }
}
// every float >= 0 by its bits, infinity included: div_refined_root on its root
__global__ void k_root(unsigned long long* bad) {
  for (unsigned long long k = blockIdx.x * blockDim.x + threadIdx.x; k <= 0x7f800000ull; k += gridDim.x * blockDim.x) {
    const float y = sqrtf(__uint_as_float((unsigned)k)), x = -__uint_as_float(0x3f800000u | (k * 2654435761u & 0x7fffffu));
    const unsigned a = __float_as_uint(div_refined(x, y)), b = __float_as_uint(div_refined_root(x, y));
    const bool nan = (a & 0x7fffffffu) > 0x7f800000u && (b & 0x7fffffffu) > 0x7f800000u;
    if (a != b && !nan) atomicAdd(bad, 1ull);
  }
}
extern "C" long check_root() {
  unsigned long long* bad = nullptr;
  unsigned long long h = ~0ull;
  if (cudaMalloc(&bad, 8) || cudaMemset(bad, 0, 8)) return -1;
  k_root<<<1184, 256>>>(bad);
  const cudaError_t e = cudaMemcpy(&h, bad, 8, cudaMemcpyDeviceToHost);
  cudaFree(bad);
  return e == cudaSuccess ? (long)h : -1;
}
extern "C" long check(unsigned first, unsigned n, int ex) {
  unsigned long long* bad = nullptr;
  unsigned long long h = ~0ull;
  if (cudaMalloc(&bad, 8) || cudaMemset(bad, 0, 8)) return -1;
  k_check<<<592, 256>>>(first, n, ex, bad);
  const cudaError_t e = cudaMemcpy(&h, bad, 8, cudaMemcpyDeviceToHost);
  cudaFree(bad);
  return e == cudaSuccess ? (long)h : -1;
}
'''


@pytest.fixture(scope="module")
def divlib(gpu, tmp_path_factory):
    d = tmp_path_factory.mktemp("div")
    cu, so = d / "t.cu", d / "t.so"
    cu.write_text(SRC)
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.check_call([nvcc, "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-I" + CSRC, "-shared",
                           "-Xcompiler", "-fPIC", "-o", str(so), str(cu)])
    lib = C.CDLL(str(so))
    lib.check.argtypes, lib.check.restype = [C.c_uint, C.c_uint, C.c_int], C.c_long
    lib.check_root.argtypes, lib.check_root.restype = [], C.c_long
    return lib


# 2^-128 is subnormal 0x00200000; 2^126 is 0x7e800000, infinity 0x7f800000
@pytest.mark.parametrize("first,n,ex", [
    (0x00200001, 0x00800000 - 0x00200001, -100), (0x00200001, 0x00800000 - 0x00200001, -20),
    (0x7e800001, 0x7f800000 - 0x7e800001, 100), (0x7e800001, 0x7f800000 - 0x7e800001, 20)])
def test_ends_of_the_range(divlib, first, n, ex):
    assert divlib.check(first, n, ex) == 0


def test_roots_need_no_more(divlib):
    """The flushing form gives div_refined's bits for the square root of every float."""
    assert divlib.check_root() == 0
