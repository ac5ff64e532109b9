"""The branch-free divisions and root of csrc/sb_math.cuh give the IEEE operations' results wherever they are used: the
logarithm and the noise radius for every 32-bit word, tanh for every float, bit for bit against the same sequences with
__fdiv_rn and __fsqrt_rn. The program is compiled here and writes nothing but its three counters."""
import os
import subprocess

import pytest

from annealing_gb300 import _build

pytestmark = pytest.mark.gpu
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "annealing_gb300", "csrc")

PROGRAM = r"""
#include <stdio.h>
#include "sb_math.cuh"

__device__ float log_ieee(float u) {
  if (!(u > 0.0f)) return -INFINITY;
  const uint32_t b = __float_as_uint(u);
  int e = (int)((b >> 23) & 0xFFu) - 127;
  float m = __uint_as_float((b & 0x007FFFFFu) | 0x3F800000u);
  if (m > 0x1.6a09e6p+0f) {
    m = __fmul_rn(m, 0.5f);
    e += 1;
  }
  const float s = __fdiv_rn(__fsub_rn(m, 1.0f), __fadd_rn(m, 1.0f));
  const float z = __fmul_rn(s, s);
  float q = __fmaf_rn(z, 0x1.c71c72p-4f, 0x1.24924ap-3f);
  q = __fmaf_rn(z, q, 0x1.99999ap-3f);
  q = __fmaf_rn(z, q, 0x1.555556p-2f);
  const float at = __fmaf_rn(__fmul_rn(s, z), q, s), fe = (float)e;
  return __fmaf_rn(fe, 0x1.62e4p-1f, __fmaf_rn(fe, 0x1.7f7d1cp-20f, __fmul_rn(2.0f, at)));
}
__device__ float tanh_ieee(float x) {
  const float ax = fabsf(x);
  if (ax != ax) return x;
  if (ax > 10.0f) return copysignf(1.0f, x);
  const float e = sbm::expm1_neg(__fmul_rn(-2.0f, ax));
  return copysignf(__fdiv_rn(-e, __fadd_rn(2.0f, e)), x);
}
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }

__global__ void compare(unsigned long long *wrong) {
  unsigned long long w[3] = {0, 0, 0};
  for (unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; k < 1ull << 32;
       k += (unsigned long long)gridDim.x * blockDim.x) {
    const float u = __fmul_rn(__uint2float_rn((uint32_t)k), 0x1p-32f);
    const float l = log_ieee(u);
    w[0] += !same(sbm::log_unit(u), l);
    w[1] += !same(sbm::root(__fmul_rn(-2.0f, sbm::log_unit(u))), __fsqrt_rn(__fmul_rn(-2.0f, l)));
    const float x = __uint_as_float((uint32_t)k);
    w[2] += !same(sbm::tanh_f(x), tanh_ieee(x));
  }
  for (int i = 0; i < 3; ++i)
    if (w[i]) atomicAdd(wrong + i, w[i]);
}

int main() {
  unsigned long long *d, h[3] = {1, 1, 1};
  if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess) return 1;
  compare<<<1024, 256>>>(d);
  if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  printf("%llu %llu %llu\n", h[0], h[1], h[2]);
  return 0;
}
"""


def test_every_input(tmp_path):
    src, exe = tmp_path / "math.cu", tmp_path / "math"
    src.write_text(PROGRAM)
    subprocess.run([_build._nvcc(), *_build.GENCODE, "-O3", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.split() == ["0", "0", "0"]
