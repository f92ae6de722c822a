// FP64 FFT of one sequence in shared memory, by one CTA, for lengths
// M = P or M = 3 P with P a power of two (the arc-length grid 6N and the
// upsampled grid N*ceil(sqrt(N)) for N = 32, 128).  Decimation in time: the
// input is split into R = M / P interleaved subsequences x[R m + r], each
// transformed by radix-2 stages (two to a pass) of length P, then combined by
// one radix-3 pass.  Bound by the FP64 pipe with many CTAs, by the latency of a
// pass with few.  Twiddles come from a table of cos/sin(2 pi j / M).
//
//   sign = -1:  X[k] = sum_n x[n] exp(-2 pi i k n / M)   (forward, unnormalised)
//   sign = +1:  X[k] = sum_n x[n] exp(+2 pi i k n / M)   (inverse, unnormalised)
#pragma once

#include <cuda_runtime.h>

__host__ __device__ inline bool ves_fft_size_ok(int M) {
  int P = (M % 3 == 0) ? M / 3 : M;
  return P >= 2 && (P & (P - 1)) == 0;
}

__device__ __forceinline__ int ves_bitrev(int v, int bits) { return (int)(__brev((unsigned)v) >> (32 - bits)); }

// x or -x by its sign bit (no FP64 instruction)
__device__ __forceinline__ double ves_signed(double x, int sign) {
  return __hiloint2double(__double2hiint(x) ^ (sign & (int)0x80000000), __double2loint(x));
}
// w (br + i bi); the products are fused in the order that the sign's constant
// folding gave before the operations were written out
__device__ __forceinline__ void ves_twiddle(double br, double bi, double wr, double wi, int sign, double& vr,
                                            double& vi) {
  vr = fma(br, wr, -(bi * wi));
  vi = sign > 0 ? fma(br, wi, bi * wr) : fma(bi, wr, br * wi);
}
// (a, b) <- (a + w b, a - w b)
__device__ __forceinline__ void ves_butterfly(double& ar, double& ai, double& br, double& bi, double wr, double wi,
                                              int sign) {
  double vr, vi;
  ves_twiddle(br, bi, wr, wi, sign, vr, vi);
  br = ar - vr;
  bi = ai - vi;
  ar = ar + vr;
  ai = ai + vi;
}

// re/im: input and output [M]; tre/tim: scratch [M]; cs/sn: cos/sin(2 pi j / (ts M)),
// j < ts M (a table of a longer length ts*M is read with stride ts).
__device__ inline void ves_fft(double* re, double* im, double* tre, double* tim, int M, const double* __restrict__ cs,
                               const double* __restrict__ sn, int sign, int ts = 1) {
  __syncthreads();
  const int R = (M % 3 == 0) ? 3 : 1;
  const int P = M / R;
  const int bits = __ffs(P) - 1;
  // scatter the R subsequences in bit-reversed order: t[r*P + rev(m)] = x[R m + r]
  for (int i = threadIdx.x; i < M; i += blockDim.x) {
    const int r = R == 3 ? i % 3 : 0, m = R == 3 ? i / 3 : i;
    const int dst = r * P + ves_bitrev(m, bits);
    tre[dst] = re[i];
    tim[dst] = im[i];
  }
  __syncthreads();
  // butterflies on each subsequence; half-size h: twiddle exp(sign 2 pi i j / (2h)).
  // Two stages at a time on four elements in registers (a single one first when
  // their number is odd): half the passes over shared memory and the barriers,
  // the same operations.
  int lh = 0;  // log2 h
  if (bits & 1) {
    for (int b = threadIdx.x; b < M / 2; b += blockDim.x) {
      double ar = tre[2 * b], ai = tim[2 * b], br = tre[2 * b + 1], bi = tim[2 * b + 1];
      ves_butterfly(ar, ai, br, bi, cs[0], ves_signed(sn[0], sign), sign);
      tre[2 * b] = ar;
      tim[2 * b] = ai;
      tre[2 * b + 1] = br;
      tim[2 * b + 1] = bi;
    }
    lh = 1;
    __syncthreads();
  }
  for (; lh < bits; lh += 2) {
    const int h = 1 << lh, st1 = ts * (M >> (lh + 1)), st2 = ts * (M >> (lh + 2));  // table steps
    for (int b = threadIdx.x; b < M / 4; b += blockDim.x) {
      const int j = b & (h - 1);
      const int i0 = ((b >> lh) << (lh + 2)) + j, i1 = i0 + h, i2 = i1 + h, i3 = i2 + h;
      double r0 = tre[i0], m0 = tim[i0], r1 = tre[i1], m1 = tim[i1];
      double r2 = tre[i2], m2 = tim[i2], r3 = tre[i3], m3 = tim[i3];
      const double wr = cs[j * st1], wi = ves_signed(sn[j * st1], sign);
      ves_butterfly(r0, m0, r1, m1, wr, wi, sign);
      ves_butterfly(r2, m2, r3, m3, wr, wi, sign);
      ves_butterfly(r0, m0, r2, m2, cs[j * st2], ves_signed(sn[j * st2], sign), sign);
      ves_butterfly(r1, m1, r3, m3, cs[(j + h) * st2], ves_signed(sn[(j + h) * st2], sign), sign);
      tre[i0] = r0;
      tim[i0] = m0;
      tre[i1] = r1;
      tim[i1] = m1;
      tre[i2] = r2;
      tim[i2] = m2;
      tre[i3] = r3;
      tim[i3] = m3;
    }
    __syncthreads();
  }
  if (R == 1) {
    for (int i = threadIdx.x; i < M; i += blockDim.x) {
      re[i] = tre[i];
      im[i] = tim[i];
    }
    __syncthreads();
    return;
  }
  // radix-3 combination: X[k + q P] = sum_r w^(r (k + q P)) X_r[k],  w = exp(sign 2 pi i / M)
  for (int k = threadIdx.x; k < P; k += blockDim.x) {
    const double x0r = tre[k], x0i = tim[k];
    const double w1r = cs[ts * k], w1i = ves_signed(sn[ts * k], sign);
    const double w2r = cs[ts * 2 * k], w2i = ves_signed(sn[ts * 2 * k], sign);
    double y1r, y1i, y2r, y2i;
    ves_twiddle(tre[P + k], tim[P + k], w1r, w1i, sign, y1r, y1i);
    ves_twiddle(tre[2 * P + k], tim[2 * P + k], w2r, w2i, sign, y2r, y2i);
    // exp(sign 2 pi i / 3) = -1/2 + sign i sqrt(3)/2
    const double c3 = -0.5, s3 = sign * 0.86602540378443864676;
    const double ar = y1r + y2r, ai = y1i + y2i;       // y1 + y2
    const double dr = y1r - y2r, di = y1i - y2i;       // y1 - y2
    re[k] = x0r + ar;
    im[k] = x0i + ai;
    // q = 1: x0 + y1 w3 + y2 w3^2 = x0 + c3 (y1 + y2) + i s3 (y1 - y2)
    re[k + P] = x0r + c3 * ar - s3 * di;
    im[k + P] = x0i + c3 * ai + s3 * dr;
    // q = 2: x0 + y1 w3^2 + y2 w3^4 = x0 + c3 (y1 + y2) - i s3 (y1 - y2)
    re[k + 2 * P] = x0r + c3 * ar + s3 * di;
    im[k + 2 * P] = x0i + c3 * ai - s3 * dr;
  }
  __syncthreads();
}
