// Shared definitions for the ves2d GB300 kernels (sm_103a).
//
// Device layout used by every kernel (vesicle-major, the transpose of the
// reference's X[2N, nv] column-per-vesicle tensors):
//   positions / densities  [nv][2][n]   (x row then y row of each vesicle)
//   tension                [nv][n]
//   per-vesicle matrices   [nv][rows][cols] row-major
//   GMRES state            [nv][3][N]   (x, y, sigma), the reference's flattening
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/ves2d_gb300.h"

#define VES_PI 3.14159265358979323846

// Device-side status word: kernels never trap; they record the first error
// code here and return.  The host reads it after the stage completes.
struct VesDeviceStatus {
  int code;      // VES_OK or a VES_ERR_* value
  int where;     // kernel-specific location tag
  long long aux; // kernel-specific detail (index that overflowed, ...)
};

__device__ __forceinline__ void ves_set_error(VesDeviceStatus* st, int code, int where, long long aux) {
  if (st == nullptr) return;
  if (atomicCAS(&st->code, VES_OK, code) == VES_OK) {
    st->where = where;
    st->aux = aux;
  }
}

template <typename T>
struct Vec2;
template <>
struct Vec2<float> {
  typedef float2 type;
};
template <>
struct Vec2<double> {
  typedef double2 type;
};

// Hardware approximate reciprocal and base-2 logarithm (MUFU), flush-to-zero.
__device__ __forceinline__ float mufu_rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float mufu_lg2(float x) {
  float r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// 1 / x for kRcpMin <= x <= kRcpMax: the hardware's approximation (within an
// ulp) and one residual step in FMA (P. Markstein, IBM J. Res. Dev. 34(1),
// 1990).  The theorem leaves out the mantissa of all ones; the result was
// compared with the division's over every mantissa and is the same
// (tests/test_gpu_arith.py).  The general division has a branch of its own
// for each call, so several of them do not overlap.
constexpr float kRcpMin = 1e-30f, kRcpMax = 1e30f;
__device__ __forceinline__ float rcp_normal(float x) {
  const float r = mufu_rcp(x);
  return fmaf(r, fmaf(-x, r, 1.0f), r);
}

// FP64 -> FP32 (to nearest even) and FP32 -> FP64 by integer operations, for
// every value with the result of the conversion.  The conversion instructions
// run on the FP64 pipe (2 lanes per clock and SM, a warp's instruction counts
// even when a predicate turns it off), integer operations at 32 times that.
__device__ __forceinline__ float narrow(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned hi = (unsigned)(b >> 32), e = (hi >> 20) & 0x7ffu, sign = hi & 0x80000000u;
  if (e - 897u <= 253u) {  // normal; the carry of 2^128 - ulp is infinity
    const unsigned long long t = b + 0x0fffffffull + ((b >> 29) & 1);
    return __uint_as_float(((unsigned)(t >> 29) - 0xC0000000u) | sign);
  }
  if (e > 1150u) return __uint_as_float(e == 0x7ffu && (b << 12) != 0 ? 0x7fffffffu : sign | 0x7f800000u);
  const int sh = e > 871u ? 926 - (int)e : 55;  // subnormal: units of 2^-149
  const unsigned long long m = (b & 0xfffffffffffffull) | (1ull << 52), q = m >> sh, rem = m - (q << sh);
  const unsigned long long half = 1ull << (sh - 1);
  return __uint_as_float(sign | ((unsigned)q + (rem > half || (rem == half && (q & 1)) ? 1u : 0u)));
}
__device__ __forceinline__ double widen(float x) {
  const unsigned b = __float_as_uint(x), a = b & 0x7fffffffu, e = a >> 23;
  unsigned hi = (a >> 3) + 0x38000000u, lo = b << 29;
  if (e - 1u > 253u) {
    if (e == 255u) {  // infinite or NaN
      hi += 0x38000000u;
    } else if (a == 0u) {
      hi = lo = 0u;
    } else {  // subnormal
      const int s = __clz((int)a) - 8;
      const unsigned m = (a << s) & 0x7fffffu;
      hi = ((unsigned)(897 - s) << 20) | (m >> 3);
      lo = m << 29;
    }
  }
  return __hiloint2double((int)((b & 0x80000000u) | hi), (int)lo);
}
__device__ __forceinline__ double widen(double x) { return x; }

// a / d with y = 1 / d from the division: a product and Markstein's correction,
// the rounding of the division (tests/test_gpu_arith.py).  What would leave the
// correction's range (exponents between -895 and 896: no intermediate result is
// subnormal), zero among it, is divided.
__device__ __forceinline__ bool mid_range(double z) {
  return (((uint32_t)__double2hiint(z) >> 20) & 0x7ffu) - 128u < 1792u;
}
__device__ __forceinline__ double quotient(double a, double d, double y) {
  const double q0 = a * y;
  const double q = fma(fma(-d, q0, a), y, q0);
  return mid_range(q) && mid_range(a) && mid_range(y) ? q : a / d;
}

// Row j of a circulant matrix (first column d) times two sequences, the matrix
// read once: sa = sum_l d[(j - l) mod n] a[l], sb with b.
__device__ __forceinline__ void circ2(const double* __restrict__ d, const double* __restrict__ a,
                                      const double* __restrict__ b, int n, int j, double& sa, double& sb) {
  double s = 0.0, t = 0.0;
  for (int l = 0; l <= j; ++l) {
    s = fma(d[j - l], a[l], s);
    t = fma(d[j - l], b[l], t);
  }
  for (int l = j + 1; l < n; ++l) {
    s = fma(d[j - l + n], a[l], s);
    t = fma(d[j - l + n], b[l], t);
  }
  sa = s;
  sb = t;
}

static inline unsigned ceil_div(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

// Host helper: map a CUDA error to a status code, recording the message.
int ves_cuda_status(cudaError_t e, const char* what);
void ves_record_error(int code, const char* fmt, ...);
