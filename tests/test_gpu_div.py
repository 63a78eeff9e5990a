"""The FP32 quotient of NewVelocity (div_rn) rounds as the division does: its
reciprocal is the rounded one for every mantissa, over the exponents its
comment names, and the quotients of 2^33 pairs agree, among them the ends of
the binade.  (With the rounded reciprocal the quotient's rounding is a theorem.)
Compiled here with the flags of the FP32 units."""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "fb_kernels.cuh"
using namespace fb;
__global__ void recips(int e, unsigned long long *bad) {
  const unsigned m = blockIdx.x * 256 + threadIdx.x;
  const float d = __uint_as_float((unsigned)(e + 127) << 23 | m);
  if (recip_rn(d) != __frcp_rn(d)) atomicAdd(bad, 1ull);
}
// n and d: mantissas of a linear congruential sequence (Knuth's), the ends of the binade in the first blocks
__global__ void quotients(unsigned long long seed, unsigned long long *bad) {
  unsigned long long x = seed + (blockIdx.x * 256ull + threadIdx.x) * 0x9E3779B97F4A7C15ull, wrong = 0;
  for (int k = 0; k < 4096; k++) {
    x = x * 6364136223846793005ull + 1442695040888963407ull;
    unsigned mn = (unsigned)(x >> 41), md = (unsigned)(x >> 18) & 0x7fffff;
    if (blockIdx.x < 64) md = md % 64 < 32 ? md % 64 : 0x7fffff - md % 64 + 32;
    const float n = __uint_as_float(0x3f800000u | mn), d = __uint_as_float(0x3f800000u | md);
    if (div_rn(n, d) != __fdiv_rn(n, d)) wrong++;
  }
  if (wrong) atomicAdd(bad, wrong);
}
extern "C" int check(unsigned long long *bad_recips, unsigned long long *bad_quotients) {
  unsigned long long *d;
  if (cudaMalloc(&d, 16) || cudaMemset(d, 0, 16)) return 1;
  for (int e = -110; e <= 110; e++) recips<<<(1 << 23) / 256, 256>>>(e, d);
  for (int r = 0; r < 32; r++) quotients<<<256, 256>>>(r + 1, d + 1);
  if (cudaMemcpy(bad_recips, d, 8, cudaMemcpyDeviceToHost) || cudaMemcpy(bad_quotients, d + 1, 8, cudaMemcpyDeviceToHost)) return 2;
  cudaFree(d);
  return 0;
}
"""


@pytest.mark.gpu
def test_div_rn_rounds_as_the_division(tmp_path):
    from fargo3d_b200 import build
    nvcc = shutil.which(build._nvcc())
    if not nvcc:
        pytest.skip("no nvcc here")
    cu, so = str(tmp_path / "div.cu"), str(tmp_path / "div.so")
    with open(cu, "w") as fh:
        fh.write(SRC)
    subprocess.run([nvcc] + build.ARCH + ["-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-prec-div=false",
                                          "-prec-sqrt=false", "-ftz=true"] + build.INC + [cu, "-o", so], check=True)
    bad = (ctypes.c_ulonglong * 2)()
    assert ctypes.CDLL(so).check(ctypes.byref(bad, 0), ctypes.byref(bad, 8)) == 0
    assert list(bad) == [0, 0]
