"""The arithmetic that kernels do in place of a CUDA operation, against that
operation: the FP32 reciprocal, the conversions by integers and the solves'
quotient have its bits, the FP64 reciprocal and logarithm from one table are
within their stated errors.

rcp_normal is compared over every mantissa, widen over every float, narrow at
every exponent with ties, their neighbours and carries; NaN only has to stay
NaN.  rcp_log states 1.3 units in the last place: next to CUDA's own error (0.5
for the division, 1 for log) that is 1.8 and 2.3 units of 2^-52 of the value."""
import json
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ves2dpy_gb300", "csrc")

SOURCE = r"""
#include <cstdio>
#include "ves_common.cuh"
#include "ves_log_table.cuh"

typedef unsigned long long u64;

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }
__device__ bool same(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b) || (a != a && b != b);
}
__device__ u64 mix(u64 x) {  // splitmix64
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}

struct Tally {  // one thread's counts, added at its end
  u64 *n, *bad, cn = 0, cb = 0;
  __device__ Tally(u64* n, u64* bad) : n(n), bad(bad) {}
  __device__ void operator()(bool ok) {
    ++cn;
    if (!ok) ++cb;
  }
  __device__ ~Tally() {
    if (cn) atomicAdd(n, cn);
    if (cb) atomicAdd(bad, cb);
  }
};

#define EACH(i, n) for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < (n); i += gridDim.x * (u64)blockDim.x)

__global__ void reciprocal(u64* n, u64* bad) {  // biased exponents 27 .. 226 hold 1e-30 .. 1e30
  Tally count(n, bad);
  EACH(i, 201ull << 23) {
    const float x = __uint_as_float((unsigned)(i + (27ull << 23)));
    if (!(x >= kRcpMin && x <= kRcpMax)) continue;
    count(same(rcp_normal(x), 1.0f / x));
  }
}
__global__ void widening(u64* n, u64* bad) {
  Tally count(n, bad);
  EACH(i, 1ull << 32) {
    const float x = __uint_as_float((unsigned)i);
    count(same(widen(x), (double)x));
  }
}
__global__ void narrowing(u64* n, u64* bad) {
  Tally count(n, bad);
  // sign, exponent, 4096 upper mantissas (the extremes among them), 8 endings
  EACH(i, 4096ull << 15) {
    const unsigned end = i & 7, top = (i >> 3) & 4095;
    const u64 se = i >> 15;
    u64 m = top == 0 ? 0 : (top == 1 ? (1ull << 52) - 1 : (top < 54 ? 1ull << (top - 2) : mix(i >> 3) >> 12));
    const u64 low = (1ull << 29) - 1;
    const u64 ends[8] = {0, 1, (1ull << 28) - 1, 1ull << 28, (1ull << 28) + 1, low, mix(i) & low, m & low};
    m = (m & ~low) | ends[end];
    const double x = __longlong_as_double((long long)((se << 52) | m));
    count(same(narrow(x), (float)x));
  }
}
__global__ void quotients(u64* n, u64* bad) {
  Tally count(n, bad);
  EACH(i, 1ull << 27) {
    u64 a = mix(2 * i), d = mix(2 * i + 1);
    const unsigned kind = i & 7;
    if (kind < 4) {  // exponents near 1
      a = (a & 0x800fffffffffffffull) | ((u64)(1003 + (a >> 52) % 41) << 52);
      d = (d & 0x800fffffffffffffull) | ((u64)(1003 + (d >> 52) % 41) << 52);
    }
    if (kind == 1) d |= 0xfffffffffffffull;                                    // mantissa of all ones
    if (kind == 2) a = (a & 0xfff0000000000000ull) | ((a >> 45) & 3);          // few bits
    if (kind == 3) d = (d & 0xfff0000000000000ull) | ((d >> 45) & 3);
    if (kind == 7 && (i & 8)) a = (i & 16) ? 0 : 0x7ff0000000000000ull;
    if (kind == 7 && (i & 32)) d = (i & 64) ? 0x8000000000000000ull : (d & 0x800fffffffffffffull);  // zero, subnormal
    const double x = __longlong_as_double((long long)a), y = __longlong_as_double((long long)d);
    count(same(quotient(x, y, 1.0 / y), x / y));
  }
}
__device__ bool log_ok(double x, const double2* tab) {
  double inv, lg;
  rcp_log(x, tab, inv, lg);
  const double ri = 1.0 / x, rl = log(x);
  const bool special = !(x >= 2.2250738585072014e-308 && x <= 1.7976931348623157e308);
  bool ok;
  if (special) {
    ok = same(inv, ri) && same(lg, rl);
  } else {
    const double u = 2.220446049250313e-16;
    const bool normal = ri >= 2.2250738585072014e-308;
    ok = (normal ? fabs(inv - ri) <= 1.8 * u * ri : same(inv, ri)) && fabs(lg - rl) <= 2.3 * u * fabs(rl);
  }
  return ok;
}
__global__ void table(u64* n, u64* bad) {
  Tally count(n, bad);
  const double2* tab = kLogTab;
  EACH(i, 2048ull * 128 * 8) {  // every exponent, around every edge of the table
    const u64 k = i & 7, e = (i >> 3) & 127, x = i >> 10;
    const u64 hm = 0x3fe6a09eull + (e << 13);
    const u64 b = ((hm << 32) + k - 4) & 0xfffffffffffffull;
    count(log_ok(__longlong_as_double((long long)((x << 52) | b)), tab));
  }
  EACH(i, 1ull << 24) count(log_ok(1.0 + ((double)i - (1 << 23)) * 1.1102230246251565e-16, tab));  // next to 1
  EACH(i, 1ull << 24) count(log_ok(1.0 + ((double)i - (1 << 23)) * 1.2e-8, tab));                  // 0.9 .. 1.1
  EACH(i, 1ull << 26) count(log_ok(__longlong_as_double((long long)mix(i)), tab));                 // any pattern
}

int main() {
  u64* c;
  cudaMallocManaged(&c, 10 * sizeof(u64));
  for (int i = 0; i < 10; ++i) c[i] = 0;
  reciprocal<<<2432, 256>>>(c, c + 1);
  widening<<<2432, 256>>>(c + 2, c + 3);
  narrowing<<<2432, 256>>>(c + 4, c + 5);
  quotients<<<2432, 256>>>(c + 6, c + 7);
  table<<<2432, 256>>>(c + 8, c + 9);
  const cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    printf("%s\n", cudaGetErrorString(e));
    return 1;
  }
  const char* name[5] = {"reciprocal", "widen", "narrow", "quotient", "rcp_log"};
  printf("{");
  for (int i = 0; i < 5; ++i) printf("%s\"%s\": [%llu, %llu]", i ? ", " : "", name[i], c[2 * i], c[2 * i + 1]);
  printf("}\n");
  return 0;
}
"""


def test_against_the_operations(tmp_path):
    from ves2dpy_gb300 import build as B
    src, exe = tmp_path / "arith.cu", tmp_path / "arith"
    src.write_text(SOURCE)
    subprocess.run([B.nvcc(), *B.ARCH, *B.FLAGS, "-I", CSRC, "-o", str(exe), str(src)], check=True, timeout=300)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout
    got = json.loads(out.stdout)
    assert all(n > 1 << 24 for n, _ in got.values()), got
    assert {k: bad for k, (_, bad) in got.items() if bad} == {}, got
