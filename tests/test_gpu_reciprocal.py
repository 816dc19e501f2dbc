"""The reciprocal of the repulsive terms (step_dev.cuh, rcp_normal) against
__fdividef(1, x) over every float that is not negative, denormal or NaN: the same
bits, so the terms are those of the reference's division by d^2 as the CUDA
documentation bounds it (zero past 2^126, a few ulps below)."""
import ctypes
import subprocess

import numpy as np
import pytest

from sop_gb300 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "step_dev.cuh"
// counts[0]: patterns compared, counts[1]: that differ; first: one that does
__global__ void compare(unsigned long long* counts, unsigned* first) {
  unsigned long long seen = 0, bad = 0;
  const unsigned all = 0x7f800000u - 0x00800000u + 1u;  // 2^-126 .. infinity
  for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < all; k += gridDim.x * blockDim.x) {
    const float x = __uint_as_float(0x00800000u + k);
    ++seen;
    if (__float_as_uint(sop::rcp_normal(x)) != __float_as_uint(__fdividef(1.0f, x))) {
      ++bad;
      *first = 0x00800000u + k;
    }
  }
  atomicAdd(counts, seen);
  atomicAdd(counts + 1, bad);
}
extern "C" int run(unsigned long long* counts, unsigned* first) {
  unsigned long long* c;
  unsigned* f;
  if (cudaMalloc(&c, 16) || cudaMalloc(&f, 4) || cudaMemset(c, 0, 16) || cudaMemset(f, 0, 4)) return 1;
  compare<<<1024, 256>>>(c, f);
  if (cudaDeviceSynchronize() || cudaMemcpy(counts, c, 16, cudaMemcpyDeviceToHost) ||
      cudaMemcpy(first, f, 4, cudaMemcpyDeviceToHost))
    return 2;
  cudaFree(c);
  cudaFree(f);
  return 0;
}
"""


def test_reciprocal_has_the_bits_of_the_approximate_division(tmp_path):
    src, so = tmp_path / "rcp.cu", tmp_path / "rcp.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", *build.ARCH,
                    "-I", build.CSRC, "-o", str(so), str(src)], check=True)
    counts, first = np.zeros(2, np.uint64), np.zeros(1, np.uint32)
    rc = ctypes.CDLL(str(so)).run(counts.ctypes.data_as(ctypes.c_void_p), first.ctypes.data_as(ctypes.c_void_p))
    assert rc == 0
    assert counts[0] == 0x7f800000 - 0x00800000 + 1
    assert counts[1] == 0, hex(first[0])
