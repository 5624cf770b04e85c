"""GPU: the arithmetic that replaces slower instructions, against those.

``widen`` and ``narrow`` (kernels.cuh) carry every FP32+IR step.  ``widen`` is
compared over all floats.  ``narrow`` is compared over doubles of every
exponent with the bit patterns at which rounding decides: zeros, halfway and
one to either side of it, carries into the next exponent, both ends of the
normal and subnormal floats, infinities and NaN, and over pseudo-random ones.

``a / over_r(b)`` must be the quotient rounded once: half an ulp, and 2^-21 of
one for the low word's two roundings (2^-24 of it each, and it is at most 2^-24
of the quotient).
"""
import ctypes
import os
import subprocess

import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "kernels.cuh"
using namespace nhw;
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }
__device__ bool same(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b) || (a != a && b != b);
}
__global__ void k_widen(unsigned long long* bad) {
  for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < 1ull << 32; i += gridDim.x * 256ull) {
    const float x = __uint_as_float((unsigned)i);
    if (!same(widen(x), (double)x)) atomicAdd(bad, 1ull);
  }
}
// mode 0: every sign and exponent, 2^16 high mantissa patterns, 16 low ones; mode 1: n hashed patterns
__global__ void k_narrow(unsigned long long* bad, int mode, unsigned long long n) {
  const unsigned long long low[16] = {0, 1, 2, 0x0fffffffull, 0x10000000ull, 0x10000001ull, 0x1fffffffull, 0x20000000ull,
                                      0x2fffffffull, 0x30000000ull, 0x30000001ull, 0x3fffffffull, 0xfffffff0ull,
                                      0xfffffff1ull, 0xefffffffull, 0xffffffffull};
  for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < n; i += gridDim.x * 256ull) {
    unsigned long long b;
    if (mode == 0) {
      const unsigned long long l = i & 15, m = (i >> 4) & 0xffff, e = i >> 20;   // e: sign and exponent
      // the two ends of the upper mantissa and what lies between, spread
      const unsigned long long hi = m < 0x100 ? m : m >= 0xff00 ? 0xf0000 | m : (m * 2654435761ull) & 0xfffff;
      b = (e << 52) | (hi << 32) | low[l];
    } else {
      b = i + 0x9e3779b97f4a7c15ull * (i + 1);
      b ^= b >> 30; b *= 0xbf58476d1ce4e5b9ull; b ^= b >> 27; b *= 0x94d049bb133111ebull; b ^= b >> 31;
      if (i & 1) b = (b & 0x800fffffffffffffull) | ((0x368ull + (b >> 52) % 0x11c) << 52);   // about the floats' range
    }
    const double x = __longlong_as_double((long long)b);
    if (!same(narrow<float>(x), (float)x)) atomicAdd(bad, 1ull);
  }
}
// quotients of hashed operands from 2^-20 to 2^20, by divisors of the same range
__global__ void k_quot(unsigned long long* bad, unsigned long long n) {
  for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < n; i += gridDim.x * 256ull) {
    unsigned long long h = 0x9e3779b97f4a7c15ull * (i + 1);
    h ^= h >> 30; h *= 0xbf58476d1ce4e5b9ull; h ^= h >> 27; h *= 0x94d049bb133111ebull; h ^= h >> 31;
    const unsigned e0 = 107 + (unsigned)(h >> 58) % 41, e1 = 107 + (unsigned)(h >> 52) % 41;
    const float a = __uint_as_float(((unsigned)h & 0x807fffffu) | e0 << 23);
    const float b = __uint_as_float(((unsigned)(h >> 24) & 0x7fffffu) | e1 << 23);
    const double exact = (double)a / (double)b, q = (double)(a / over_r<float>(b));
    const double ulp = ldexp(1.0, ilogb(exact) - 23);
    if (!(fabs(q - exact) <= (0.5 + 0x1p-21) * ulp)) atomicAdd(bad, 1ull);
  }
}
extern "C" long long mismatches(int what) {
  unsigned long long* bad = nullptr;
  unsigned long long h = ~0ull;
  if (cudaMalloc((void**)&bad, 8) != cudaSuccess || cudaMemset(bad, 0, 8) != cudaSuccess) return -1;
  if (what == 0) k_widen<<<152 * 8, 256>>>(bad);
  else if (what < 3) k_narrow<<<152 * 8, 256>>>(bad, what - 1, 1ull << 32);
  else k_quot<<<152 * 8, 256>>>(bad, 1ull << 28);
  if (cudaMemcpy(&h, bad, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  cudaFree(bad);
  return (long long)h;
}
"""


@pytest.fixture(scope="module")
def compiled(tmp_path_factory):
    from nhwave_gb300 import build
    d = tmp_path_factory.mktemp("conv")
    src, so = d / "conv.cu", d / "libconv.so"
    src.write_text(SOURCE)
    subprocess.check_call([build._nvcc(), "-std=c++17", "-O3", "--extended-lambda", "--fmad=true", *build.ARCH, "-shared",
                           "-Xcompiler", "-fPIC", "-I", os.path.join(REPO, "nhwave_gb300", "csrc"), str(src), "-o",
                           str(so)])
    lib = ctypes.CDLL(str(so))
    lib.mismatches.restype = ctypes.c_longlong
    return lib


@pytest.mark.parametrize("what", [0, 1, 2, 3], ids=["widen_all", "narrow_edges", "narrow_random", "quotients"])
def test_conversions_equal_the_instructions(what, compiled):
    assert compiled.mismatches(what) == 0
