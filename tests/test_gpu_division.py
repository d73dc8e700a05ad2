"""The branch-free reciprocal and quotients of the FP64 forms (rcp_mk, div_mk, div_mk2)
against CUDA's correctly rounded __drcp_rn and __ddiv_rn, bit for bit, over random operands
of the whole range they take: both ends of mk_range, significands near all ones and near
powers of two, low words of all ones.  The device functions are compiled from their header
into a small library of this test's own."""
import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "sw-mpdec_b200", "csrc")

SOURCE = r"""
#include "swm_device.cuh"
using namespace swm;

__device__ unsigned long long draw(unsigned long long& s) {  // xorshift64*
  s ^= s << 13;
  s ^= s >> 7;
  s ^= s << 17;
  return s * 0x2545F4914F6CDD1Dull;
}
__device__ bool same(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}
// out: [tested, reciprocals, div_mk, div_mk2, div_rn, mk_plain, mk_range] mismatches
__global__ void check(unsigned long long seed, int n, int pattern, unsigned long long* out) {
  unsigned long long s =
      seed + (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) * 0x9E3779B97F4A7C15ull;
  if (s == 0) s = 1;
  const unsigned long long frac = (1ull << 52) - 1;
  unsigned long long bad[7] = {};
  for (int i = 0; i < n; ++i) {
    unsigned long long my = draw(s) & frac, mx = draw(s) & frac;
    const unsigned long long a = draw(s), b = draw(s), keep = draw(s) % 53;
    switch (pattern) {
      case 1: my |= frac >> keep; break;                  // low bits ones
      case 2: my |= frac & ~((1ull << keep) - 1); break;  // high bits ones
      case 3: my &= (1ull << keep) - 1; break;            // near a power of two from above
      case 4: my |= 0xffffffffull; break;                 // low word all ones
      case 5: my = frac; break;                           // all ones
      default: break;
    }
    if (a & 1) mx = mx | (frac & ~((1ull << keep) - 1));
    // exponents of [2^-400, 2^400), its two ends every fourth draw
    unsigned long long ey = 623 + (a >> 8) % 800, ex = 623 + (b >> 8) % 800;
    if ((a & 12) == 4) ey = (a & 16) ? 623 : 1422;
    if ((b & 12) == 4) ex = (b & 16) ? 623 : 1422;
    const double y = __longlong_as_double((long long)(my | (ey << 52) | ((a & 2) << 62)));
    const double x = __longlong_as_double((long long)(mx | (ex << 52) | ((b & 2) << 62)));
    ++bad[0];
    const double r = __drcp_rn(y), q = __ddiv_rn(x, y);
    if (mk_plain(y) && my == frac) ++bad[5];
    if (!mk_range(x) || !mk_range(y)) ++bad[6];
    if (mk_plain(y)) {
      const double rm = rcp_mk(y);
      if (!same(rm, r)) ++bad[1];
      if (!same(div_mk2(x, y, rm, mk_low(y, rm)), q)) ++bad[3];
    }
    if (!same(div_mk(x, y, r), q)) ++bad[2];
    if (!same(div_rn(x, y, r), q)) ++bad[4];
    // just outside the range, and anything at all through div_rn
    const double lo = __longlong_as_double((long long)(my | (622ull << 52)));
    const double hi = __longlong_as_double((long long)(my | (1423ull << 52)));
    if (mk_range(lo) || mk_range(hi) || mk_range(0.) || mk_range(y / 0.)) ++bad[6];
    const double u = __longlong_as_double((long long)a), v = __longlong_as_double((long long)b);
    const double w = __ddiv_rn(u, v);
    if (!same(div_rn(u, v, __drcp_rn(v)), w) && !(w != w)) ++bad[4];
  }
  for (int k = 0; k < 7; ++k) atomicAdd(&out[k], bad[k]);
}
extern "C" int run(unsigned long long seed, int n, int pattern, unsigned long long* out) {
  unsigned long long* d;
  if (cudaMalloc(&d, 56)) return 1;
  cudaMemset(d, 0, 56);
  check<<<148 * 8, 256>>>(seed, n, pattern, d);
  const cudaError_t e = cudaMemcpy(out, d, 56, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    import build
    d = tmp_path_factory.mktemp("division")
    src, so = str(d / "division.cu"), str(d / "division.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([build.NVCC, *build.ARCH, "-O3", "-std=c++17", "-fmad=false", "-I", CSRC,
                    "-shared", "-Xcompiler", "-fPIC", src, "-o", so], check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("pattern", range(6))
def test_equal_to_the_correctly_rounded_operations(gpu, lib, pattern):
    out = (ctypes.c_ulonglong * 7)()
    assert lib.run(ctypes.c_ulonglong(20260 + pattern), 500, pattern, out) == 0
    tested, *bad = out
    assert tested == 148 * 8 * 256 * 500
    assert bad == [0] * 6
