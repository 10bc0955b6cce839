"""The box means' quotient (csrc/window.cuh, SoftDiv) against the device's own division, bit for bit: every window length
from 1 to 2001 with every significand, at the smallest and at ordinary exponents, with every subnormal, and infinities
and NaN.  (A negative zero may come back as a positive one; it is not tried.)"""
import ctypes
import os
import subprocess

import pytest

SOURCE = """
#include "window.cuh"
using namespace hdog;

// blockIdx.y: the length 2 y + 1; a: significand i at the exponent of `base`'s bits (i counts up from them)
__global__ void compare(unsigned base, unsigned n, unsigned long long *wrong) {
  const unsigned i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const int len = 2 * blockIdx.y + 1;
  const SoftDiv div(len);
  const float a = __uint_as_float(base + i), want = __fdiv_rn(a, (float)len);
  const float2 got = div(make_float2(a, -a));
  const bool nan = want != want;
  const bool same = nan ? got.x != got.x && got.y != got.y
                        : __float_as_uint(got.x) == __float_as_uint(want) &&
                              (a == 0.0f || __float_as_uint(got.y) == __float_as_uint(-want));
  if (!same) atomicAdd(wrong, 1ull);
}

extern "C" long long run(unsigned base, unsigned n) {
  unsigned long long *wrong = nullptr, host = ~0ull;
  if (cudaMalloc(&wrong, 8) != cudaSuccess) return -1;
  cudaMemset(wrong, 0, 8);
  compare<<<dim3((n + 255) / 256, 1001), 256>>>(base, n, wrong);
  if (cudaDeviceSynchronize() != cudaSuccess) return -2;
  cudaMemcpy(&host, wrong, 8, cudaMemcpyDeviceToHost);
  cudaFree(wrong);
  return (long long)host;
}
"""


@pytest.mark.gpu
def test_gpu_quotients_equal_the_division(tmp_path):
    import hdog
    src, so = str(tmp_path / "d.cu"), str(tmp_path / "d.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    r = subprocess.run(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-shared", "-Xcompiler",
                        "-fPIC", "-I", os.path.join(hdog._PKG, "csrc"), "-I",
                        os.path.join(os.path.dirname(hdog._PKG), "include"), src, "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(so)
    lib.run.restype, lib.run.argtypes = ctypes.c_longlong, [ctypes.c_uint, ctypes.c_uint]
    mantissas = 1 << 23
    assert lib.run(0, mantissas) == 0                      # zero and the subnormals
    for exponent in (1, 12, 126, 127, 200, 254):           # the smallest normals: quotients among the subnormals
        assert lib.run(exponent << 23, mantissas) == 0, exponent
    assert lib.run(255 << 23, 4) == 0                      # infinity and NaN
