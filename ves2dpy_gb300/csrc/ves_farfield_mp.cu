// All-pairs Stokeslet sum (allExactStokesSLTarget_compare1/2,
// mytorch/biem_support.py:7-272; Poten.exactStokesSL, mytorch/poten.py:280-336)
// evaluated with a multipole expansion of each source vesicle for the
// vesicle pairs that are well separated, and by the direct FP32 sum for the
// others (precision VES_PREC_FP32M).
//
// The sum is the reference's: for a target x and a source vesicle with
// upsampled points w_j and quadrature-weighted densities f_j (complex
// notation, f = fx + i fy),
//
//   u(x) = sum_j [ -1/2 log|r_j|^2 f_j + (r_j . f_j) r_j / |r_j|^2 ],  r_j = x - w_j
//        = sum_j [ -1/2 log|r_j|^2 f_j + 1/2 f_j + 1/2 conj(f_j) r_j / conj(r_j) ].
//
// With the source centre c, v_j = w_j - c, omega = x - c, R >= max |v_j|,
// normalised vt_j = v_j / R and tau = R / omega (|tau| = rho < 1):
//
//   u = -log|omega| F0 + F0/2 + sum_{k>=1} [tau^k A_k + conj(tau)^k B_k] / (2k)
//       + 1/2 (omega / conj(omega)) conj(sum_{k>=0} tau^k A_k)
//       - 1/2 conj(tau sum_{k>=0} tau^k E_k)
//
//   F0 = sum f_j,  A_k = sum f_j vt_j^k,  B_k = sum f_j conj(vt_j)^k,
//   E_k = sum f_j conj(vt_j) vt_j^k
//
// (series of log(1 - v/omega) and 1/(1 - conj(v/omega))).  Truncating at
// order P leaves at most sum_j |f_j| rho^(P+1) / (1 - rho) per series.  A
// (target vesicle, source vesicle) pair uses the expansion when
// rho_pair = R_s / (|c_t - c_s| - R_t) <= kRhoMax, with P the smallest order
// whose bound is below kEps (relative to sum |f_j|); every other pair, every
// pair on the target's near-candidate list (where single target points are
// excluded, biem_support.py:218-219), is summed directly over the
// upsampled points in FP32 with the source-centred logarithm of the FP32C
// path.  The moments are sums over exactly the upsampled points of the direct
// rule (centre, radius and F0 in FP64, the others in FP32, stored in FP32);
// the series are evaluated in FP32 (Horner) and the per-source contributions
// are added with Neumaier compensation.
#include "ves_internal.h"
#include "ves_tc.cuh"

namespace {

constexpr int kPMax = 24;                 // highest expansion order
constexpr float kRhoMax = 0.35f;          // 0.35^25 / 0.65 < 1e-11
constexpr float kEps = 1e-10f;            // truncation bound relative to sum |f_j|
constexpr int kStage = 32;                // source vesicles per shared-memory stage
constexpr int kLow = 13;                  // orders 0 .. kLow - 1 of a source are staged, the others read from L2
constexpr double kHalfLn2 = 0.34657359027997264;

struct __align__(16) MPSrc {
  float2 chi, clo;  // centre, high and low FP32 parts
  float2 f0;        // sum of the density
  float R;          // bound on |w_j - c| over the upsampled points
  float pad;
};

// one order k of one source: Al = A_k/(2k) (0 at k=0), Bc = conj(B_k/(2k))
// (0 at k=0), A_k, E_k, the real and the imaginary parts of (Al, Bc) and of
// (A, E) side by side, as the packed FP32x2 Horner steps take them
struct __align__(16) MPMom {
  float2 abr, abi, aer, aei;
};
// order k of source s: the low orders of every source come first, so that a
// stage of sources is one contiguous copy
__host__ __device__ inline long long mom_at(int nsrc, int s, int k) {
  return k < kLow ? (long long)s * kLow + k : (long long)nsrc * kLow + (long long)s * (kPMax + 1 - kLow) + (k - kLow);
}

__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}

// ---------------------------------------------------------------------------
// One CTA (256 threads) per source vesicle: centre, FP32 records for the
// direct rule, density sum, radius bound and the normalised moments.
__global__ void __launch_bounds__(256) mp_prep_kernel(int ns, const double* __restrict__ X,
                                                      const double* __restrict__ den, float4* __restrict__ rec,
                                                      MPSrc* __restrict__ src, MPMom* __restrict__ mom) {
  __shared__ double red[3][256];
  __shared__ float4 pts[256];  // (v, f) of 256 points
  const int s = blockIdx.x, t = threadIdx.x;
  const double* x = X + (long long)s * 2 * ns;
  const double* f = den + (long long)s * 2 * ns;
  double sx = 0, sy = 0;
  for (int j = t; j < ns; j += 256) {
    sx += x[j];
    sy += x[ns + j];
  }
  red[0][t] = sx;
  red[1][t] = sy;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (t < w) {
      red[0][t] += red[0][t + w];
      red[1][t] += red[1][t + w];
    }
    __syncthreads();
  }
  const double cx = red[0][0] / ns, cy = red[1][0] / ns;
  __syncthreads();
  double r2 = 0, fx = 0, fy = 0;
  for (int j = t; j < ns; j += 256) {
    const double lx = x[j] - cx, ly = x[ns + j] - cy;
    rec[(long long)s * ns + j] = make_float4((float)lx, (float)ly, (float)f[j], (float)f[ns + j]);
    r2 = fmax(r2, lx * lx + ly * ly);
    fx += f[j];
    fy += f[ns + j];
  }
  red[0][t] = r2;
  red[1][t] = fx;
  red[2][t] = fy;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (t < w) {
      red[0][t] = fmax(red[0][t], red[0][t + w]);
      red[1][t] += red[1][t + w];
      red[2][t] += red[2][t + w];
    }
    __syncthreads();
  }
  double R = sqrt(red[0][0]) * (1.0 + 1e-6);
  if (!(R > 0)) R = 1.0;
  if (t == 0) {
    MPSrc o;
    o.chi = make_float2((float)cx, (float)cy);
    o.clo = make_float2((float)(cx - (double)o.chi.x), (float)(cy - (double)o.chi.y));
    o.f0 = make_float2((float)red[1][0], (float)red[2][0]);
    o.R = (float)R;
    o.pad = 0.f;
    src[s] = o;
  }
  // moments: warp w takes orders k = w, w + 8, w + 16, ... (<= kPMax); lanes
  // split the points.  FP32 sums: a moment of order k enters the series
  // multiplied by rho^k and is stored in FP32, so FP32 accumulation (errors
  // of a few 1e-8 of sum |f| |v|^k) matches the storage; the monopole F0 is
  // the FP64 density sum above.
  const int warp = t >> 5, lane = t & 31;
  constexpr int kPer = (kPMax + 8) / 8;  // orders per warp
  float2 A[kPer], B[kPer], E[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) A[q] = B[q] = E[q] = make_float2(0.f, 0.f);
  const double iR = 1.0 / R;
  for (int c0 = 0; c0 < ns; c0 += 256) {
    // each point scaled once (FP64 is the slow pipe) and read by every warp:
    // 262 -> 122 us at 1024 x N=128
    __syncthreads();
    if (c0 + t < ns) {
      const int j = c0 + t;
      pts[t] = make_float4((float)((x[j] - cx) * iR), (float)((x[ns + j] - cy) * iR), (float)f[j], (float)f[ns + j]);
    }
    __syncthreads();
    for (int j = lane; j < min(256, ns - c0); j += 32) {
      const float4 pt = pts[j];
      const float2 v = make_float2(pt.x, pt.y);
      const float2 fj = make_float2(pt.z, pt.w);
      float2 pw = make_float2(1.f, 0.f), v8 = v;  // pw = v^warp, v8 = v^8
      for (int e = 0; e < warp; ++e) pw = cmulf(pw, v);
      v8 = cmulf(v8, v8);
      v8 = cmulf(v8, v8);
      v8 = cmulf(v8, v8);
      const float2 fvb = cmulf(fj, make_float2(v.x, -v.y));  // f conj(v)
#pragma unroll
      for (int q = 0; q < kPer; ++q) {
        if (warp + 8 * q > kPMax) break;
        const float2 a = cmulf(fj, pw);
        const float2 b = cmulf(fj, make_float2(pw.x, -pw.y));
        const float2 e = cmulf(fvb, pw);
        A[q].x += a.x;
        A[q].y += a.y;
        B[q].x += b.x;
        B[q].y += b.y;
        E[q].x += e.x;
        E[q].y += e.y;
        pw = cmulf(pw, v8);
      }
    }
  }
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    for (int o = 16; o > 0; o >>= 1) {
      A[q].x += __shfl_xor_sync(0xffffffffu, A[q].x, o);
      A[q].y += __shfl_xor_sync(0xffffffffu, A[q].y, o);
      B[q].x += __shfl_xor_sync(0xffffffffu, B[q].x, o);
      B[q].y += __shfl_xor_sync(0xffffffffu, B[q].y, o);
      E[q].x += __shfl_xor_sync(0xffffffffu, E[q].x, o);
      E[q].y += __shfl_xor_sync(0xffffffffu, E[q].y, o);
    }
    const int k = warp + 8 * q;
    if (lane == 0 && k <= kPMax) {
      MPMom m;
      const float h = k > 0 ? 0.5f / k : 0.f;
      const float2 ac = k > 0 ? A[q] : make_float2((float)red[1][0], (float)red[2][0]);  // A_0 = F0 (FP64 sum)
      m.abr = make_float2(A[q].x * h, B[q].x * h);
      m.abi = make_float2(A[q].y * h, -B[q].y * h);
      m.aer = make_float2(ac.x, E[q].x);
      m.aei = make_float2(ac.y, E[q].y);
      mom[mom_at(gridDim.x, s, k)] = m;
    }
  }
}

// target vesicles: centre (hi/lo) and FP32 local coordinates
__global__ void __launch_bounds__(256) mp_prep_targets_kernel(int ntp, const double* __restrict__ X,
                                                              float2* __restrict__ local, float2* __restrict__ chi,
                                                              float2* __restrict__ clo) {
  __shared__ double red[2][256];
  const int k = blockIdx.x, t = threadIdx.x;
  const double* x = X + (long long)k * 2 * ntp;
  double sx = 0, sy = 0;
  for (int j = t; j < ntp; j += 256) {
    sx += x[j];
    sy += x[ntp + j];
  }
  red[0][t] = sx;
  red[1][t] = sy;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (t < w) {
      red[0][t] += red[0][t + w];
      red[1][t] += red[1][t + w];
    }
    __syncthreads();
  }
  const double cx = red[0][0] / ntp, cy = red[1][0] / ntp;
  for (int j = t; j < ntp; j += 256) local[(long long)k * ntp + j] = make_float2((float)(x[j] - cx), (float)(x[ntp + j] - cy));
  if (t == 0) {
    const float hx = (float)cx, hy = (float)cy;
    chi[k] = make_float2(hx, hy);
    clo[k] = make_float2((float)(cx - (double)hx), (float)(cy - (double)hy));
  }
}

// One source set (the upsampled points of one group of vesicles).
struct MPSet {
  int nsrc, ns;
  const float4* rec;  // [nsrc][ns] direct-rule records
  const MPSrc* src;   // [nsrc]
  const MPMom* mom;   // moments, see mom_at
};

constexpr int kMPSets = 4;

struct MPGroupArgs {
  int ng;
  MPSet set[kMPSets];            // source sets
  int cta0[kMPSets + 1];         // first CTA of each target set
  int upc[kMPSets];              // warps' worth of points (units) per target column
  int nt[kMPSets], ntp[kMPSets];
  const float2* tloc[kMPSets];   // [nt][ntp] per target set
  const float2* thi[kMPSets];
  const float2* tlo[kMPSets];
  double* out[kMPSets];          // [nt][2][ntp] per target set, scaled by 1/(4 pi)
  const int* self_idx[kMPSets];  // source index (in the same set) of each column's own vesicle; null: see own
  int own[kMPSets];              // without self_idx: 1: column = source index, 0: no own vesicle
  // near lists of target set g against source set q, [g][q]: ascending source indices
  const int* cand_count[kMPSets][kMPSets];
  const int* cand_src[kMPSets][kMPSets];
  const uint32_t* excl_mask[kMPSets][kMPSets];
  int maxc[kMPSets][kMPSets];
  int nwords[kMPSets];
  unsigned long long* work;      // optional: series terms, direct pairs (per target point)
  VesDeviceStatus* st;
};

// Every pair of a stage as one lane of the warp sees it: target centre
// relative to the source's (hi/lo: no cancellation from absolute positions)
// and what to do: order P >= 1 of the expansion, 0: the target's own vesicle,
// < 0: direct rule (-1, or -2 - place on the near list).
struct __align__(16) MPPair {
  float ox, oy, R;
  int code;
};

// Compensated addition of one source's contribution to (x, y) totals; the
// error term of the rounded sum is exact (Knuth's TwoSum).
__device__ __forceinline__ void two_sum(float2& tot, float2& cmp, float2 v) {
  const float2 m1 = make_float2(-1.f, -1.f);  // a - b as fma(b, -1, a): the same rounding
  const float2 t = __fadd2_rn(tot, v);
  const float2 z = __ffma2_rn(tot, m1, t);
  const float2 a = __ffma2_rn(__ffma2_rn(z, m1, t), m1, tot), b = __ffma2_rn(z, m1, v);
  cmp = __fadd2_rn(cmp, __fadd2_rn(a, b));
  tot = t;
}

// One Horner step of the four series, two to a packed FP32x2 register pair
// (A/2k with conj B/2k, A with E): h = h tau + m.  u = (ur, ur), w = (ui, ui),
// mw = (-ui, -ui).
__device__ __forceinline__ void horner(float2& xr, float2& xi, float2& yr, float2& yi, const MPMom& m, float2 u,
                                       float2 w, float2 mw) {
  const float2 a = __ffma2_rn(xr, u, __ffma2_rn(xi, mw, m.abr));
  xi = __ffma2_rn(xr, w, __ffma2_rn(xi, u, m.abi));
  xr = a;
  const float2 b = __ffma2_rn(yr, u, __ffma2_rn(yi, mw, m.aer));
  yi = __ffma2_rn(yr, w, __ffma2_rn(yi, u, m.aei));
  yr = b;
}

// Sum over the sources of every set onto the target points of every set.
//
// Bound by instruction issue: 16 fma per series term (about 6 terms per
// separated pair) and ~60 operations more per pair.  A warp owns 32 points of
// one target column (one unit); the warps of a CTA share the staged sources
// (kLow orders of 32 bytes and one record each, by bulk copy, two stages in
// flight).  What depends on the pair of vesicles alone (offset, order of the
// expansion, place on the near list) is worked out once per warp, one source
// per lane, and read back as a broadcast; the four complex Horner recurrences
// run as packed FP32x2 fmas, two series to a register pair, which halves the
// instructions per term.  Close pairs run the direct rule on records staged
// 32 at a time by the warp itself, so no warp waits for another's close pairs
// inside a stage, and a stage's buffer is refilled by the warp that leaves it
// last, so that none waits for another's between stages either (S == 1).  Five
// CTAs of four warps per SM (102 registers): with 80 registers the direct
// rule's loads and MUFU results are not overlapped, with 128 the series wait.
// One sum: 8192 x N=32 32.6 -> 12.9 ms, 4096 x N=128 20.7 -> 14.9, 1024 x N=128
// 2.44 -> 2.00, 333 x N=64 0.49 -> 0.23.
//
// S warps share one unit when there are too few units to fill the chip: they
// take the sources of a stage in turn and leave the contributions in shared
// memory, where the unit's first warp adds them in source order.  A point's
// contributions are always added in source order, so the result does not
// depend on S.
template <int WARPS, int S>
__global__ void __launch_bounds__(WARPS * 32, S == 1 ? 5 : 16 / WARPS) mp_eval_kernel(MPGroupArgs p) {
  constexpr int kUnits = WARPS / S;
  __shared__ __align__(128) MPMom smom[2][kStage * kLow];
  __shared__ __align__(16) MPSrc ssrc[2][kStage];
  __shared__ MPPair pairs[WARPS][kStage];
  __shared__ float4 drec[WARPS][32];
  __shared__ float2 part[S > 1 ? 2 : 1][S > 1 ? kUnits : 1][S > 1 ? kStage : 1][32];
  __shared__ int turn[2][kUnits], done[2];
  __shared__ uint64_t bar[2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int unit = warp / S, sub = warp % S;
  int g = 0;
  while (g + 1 < p.ng && (int)blockIdx.x >= p.cta0[g + 1]) ++g;
  const int ntp = p.ntp[g], upc = p.upc[g];
  const long long u = (long long)(blockIdx.x - p.cta0[g]) * kUnits + unit;
  const bool live = u < (long long)p.nt[g] * upc;
  const int col = live ? (int)(u / upc) : 0;
  const int i = (live ? (int)(u % upc) : 0) * 32 + lane;
  const bool valid = live && i < ntp;
  const float2* tl_col = p.tloc[g] + (long long)col * ntp;
  const float2 tl = valid ? tl_col[i] : make_float2(0.f, 0.f);
  const float2 thi = p.thi[g][col], tlo = p.tlo[g][col];
  // radius of the target vesicle about its centre
  float RT = 0.f;
  for (int k = lane; k < ntp; k += 32) {
    const float2 t = tl_col[k];
    RT = fmaxf(RT, sqrtf(t.x * t.x + t.y * t.y));
  }
  for (int o = 16; o > 0; o >>= 1) RT = fmaxf(RT, __shfl_xor_sync(0xffffffffu, RT, o));
  RT = RT * (1.0f + 1e-6f);
  if (threadIdx.x == 0) {
    tc_mbar_init(&bar[0], 1);
    tc_mbar_init(&bar[1], 1);
    tc_mbar_fence_init();
    tc_fence_async_smem();
  }
  if (threadIdx.x < 2 * kUnits) turn[threadIdx.x / kUnits][threadIdx.x % kUnits] = 0;
  if (threadIdx.x < 2) done[threadIdx.x] = 0;
  __syncthreads();
  float2 tot = make_float2(0.f, 0.f), cmp = make_float2(0.f, 0.f);
  unsigned terms = 0, ndirect = 0;
  int kst = 0;  // stages so far: stage buffers and barrier phases alternate
  bool failed = false;
  for (int q = 0; q < p.ng; ++q) {
    // every warp is through with the last set's stages, or one has given up
    if (q > 0 && __syncthreads_or(failed ? 1 : 0)) break;
    const MPSet& set = p.set[q];
    const int nstages = (set.nsrc + kStage - 1) / kStage;
    auto fetch = [&](int st, int buf) {  // thread 0
      const int s0 = st * kStage, n = min(kStage, set.nsrc - s0);
      tc_expect_tx(&bar[buf], (uint32_t)(n * (kLow * sizeof(MPMom) + sizeof(MPSrc))));
      tc_bulk_g2s(smom[buf], set.mom + (long long)s0 * kLow, (uint32_t)(n * kLow * sizeof(MPMom)), &bar[buf]);
      tc_bulk_g2s(ssrc[buf], set.src + s0, (uint32_t)(n * sizeof(MPSrc)), &bar[buf]);
    };
    if (threadIdx.x == 0)
      for (int st = 0; st < 2 && st < nstages; ++st) fetch(st, (kst + st) & 1);
    const int self = q != g ? -1 : (p.self_idx[g] ? p.self_idx[g][col] : (p.own[g] ? col : -1));
    const int mc = p.maxc[g][q];
    const int cend = p.cand_count[g][q] ? min(p.cand_count[g][q][col], mc) : 0;
    const int* cands = p.cand_src[g][q] ? p.cand_src[g][q] + (long long)col * mc : nullptr;
    const uint32_t* excl = p.excl_mask[g][q] ? p.excl_mask[g][q] + (long long)col * mc * p.nwords[g] : nullptr;
    for (int st = 0; st < nstages; ++st, ++kst) {
      const int buf = kst & 1, s0 = st * kStage, n = min(kStage, set.nsrc - s0);
      if (!tc_mbar_wait(&bar[buf], (kst >> 1) & 1, p.st, 30)) failed = true;
      __syncwarp();  // S == 1: the previous stage's pairs have been read
      if (lane < n) {
        const MPSrc Sq = ssrc[buf][lane];
        const int s = s0 + lane;
        const float ox = (thi.x - Sq.chi.x) + (tlo.x - Sq.clo.x);
        const float oy = (thi.y - Sq.chi.y) + (tlo.y - Sq.clo.y);
        int lo = 0, hi = cend;  // first candidate >= s
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (cands[mid] < s) lo = mid + 1; else hi = mid;
        }
        const bool cand = lo < cend && cands[lo] == s;
        const float dc = sqrtf(ox * ox + oy * oy) - RT;
        const float rp = dc > 0.f ? Sq.R / dc : 2.f;
        int code;
        if (s == self) {
          code = 0;
        } else if (!cand && rp <= kRhoMax) {
          // expansion of order P: rp^(P+1) / (1 - rp) <= kEps
          const int P = rp > 0.f ? (int)ceilf(__logf(kEps * (1.f - rp)) / __logf(rp)) - 1 : 1;
          code = max(1, min(P, kPMax));
        } else {
          code = cand ? -2 - lo : -1;
        }
        if (p.work && live && sub == 0) {
          terms += code > 0 ? code + 1 : 0;
          ndirect += code < 0 ? set.ns : 0;
        }
        pairs[warp][lane] = MPPair{ox, oy, Sq.R, code};
      }
      __syncwarp();
      for (int qs = 0;; ++qs) {
        if (S > 1) {  // the unit's warps take the stage's sources in turn
          if (lane == 0) qs = atomicAdd(&turn[buf][unit], 1);
          qs = __shfl_sync(0xffffffffu, qs, 0);
        }
        if (qs >= n || !live) break;
        const MPPair pr = pairs[warp][qs];
        float2 v = make_float2(0.f, 0.f);
        if (pr.code > 0) {
          const float tx = tl.x + pr.ox, ty = tl.y + pr.oy;  // omega
          const float om2 = fmaf(tx, tx, ty * ty);
          const float iom2 = mufu_rcp(om2);
          const float ur = pr.R * tx * iom2, ui = -pr.R * ty * iom2;  // tau = R / omega
          const float2 uu = make_float2(ur, ur), ww = make_float2(ui, ui), mw = make_float2(-ui, -ui);
          const MPMom* m = smom[buf] + qs * kLow;
          float2 xr, xi, yr, yi;
          int k = pr.code;
          if (k >= kLow) {  // the few orders past the staged ones
            const MPMom* hm = set.mom + mom_at(set.nsrc, s0 + qs, kLow);
            const MPMom t = hm[k - kLow];
            xr = t.abr, xi = t.abi, yr = t.aer, yi = t.aei;
            for (--k; k >= kLow; --k) horner(xr, xi, yr, yi, hm[k - kLow], uu, ww, mw);
            ++k;
          } else {
            const MPMom t = m[k];
            xr = t.abr, xi = t.abi, yr = t.aer, yi = t.aei;
          }
          switch (k) {  // orders k - 1 .. 0, straight-line
#define VES_MP_STEP(K) case K + 1: horner(xr, xi, yr, yi, m[K], uu, ww, mw);
            VES_MP_STEP(12) VES_MP_STEP(11) VES_MP_STEP(10) VES_MP_STEP(9) VES_MP_STEP(8) VES_MP_STEP(7)
            VES_MP_STEP(6) VES_MP_STEP(5) VES_MP_STEP(4) VES_MP_STEP(3) VES_MP_STEP(2) VES_MP_STEP(1) VES_MP_STEP(0)
#undef VES_MP_STEP
            default: break;
          }
          const float2 f0 = ssrc[buf][qs].f0;
          const float lnom = (float)kHalfLn2 * mufu_lg2(om2);  // log|omega|
          // (omega / conj(omega)) conj(hC) and conj(tau hE)
          const float qr = (tx * tx - ty * ty) * iom2, qi = 2.f * tx * ty * iom2;
          const float wcr = qr * yr.x + qi * yi.x, wci = qi * yr.x - qr * yi.x;
          const float ter = ur * yr.y - ui * yi.y, tei = -(ur * yi.y + ui * yr.y);
          v.x = fmaf(-lnom, f0.x, 0.5f * f0.x) + xr.x + xr.y + 0.5f * (wcr - ter);
          v.y = fmaf(-lnom, f0.y, 0.5f * f0.y) + xi.x - xi.y + 0.5f * (wci - tei);
        } else if (pr.code < 0) {
          // direct rule over the upsampled points (FP32, log relative to the source centre)
          const float4* R4 = set.rec + (long long)(s0 + qs) * set.ns;
          bool ex = false;
          if (pr.code < -1 && valid) {
            const uint32_t w = excl[(long long)(-2 - pr.code) * p.nwords[g] + (i >> 5)];
            ex = (w >> (i & 31)) & 1u;
          }
          const float tx = tl.x + pr.ox, ty = tl.y + pr.oy;
          const float rc2 = fmaf(tx, tx, ty * ty);
          const float irc2 = mufu_rcp(rc2);
          float2 ac = make_float2(0.f, 0.f), al = make_float2(0.f, 0.f);
          float4 nx = lane < set.ns ? R4[lane] : make_float4(0.f, 0.f, 0.f, 0.f);
          for (int j0 = 0; j0 < set.ns; j0 += 32) {
            __syncwarp();
            drec[warp][lane] = nx;
            __syncwarp();
            if (j0 + 32 + lane < set.ns) nx = R4[j0 + 32 + lane];
            const int nj = min(32, set.ns - j0);
#pragma unroll 8
            for (int j = 0; j < nj; ++j) {
              const float4 r = drec[warp][j];
              const float dx = tx - r.x, dy = ty - r.y;
              const float r2 = fmaf(dx, dx, dy * dy);
              const float inv = mufu_rcp(r2);
              const float lg = mufu_lg2(r2 * irc2);
              const float cc = fmaf(dx, r.z, dy * r.w) * inv;
              ac = __ffma2_rn(make_float2(cc, cc), make_float2(dx, dy), ac);
              al = __ffma2_rn(make_float2(lg, lg), make_float2(r.z, r.w), al);
            }
          }
          if (!ex) {
            const float2 f0 = ssrc[buf][qs].f0;
            const float lgc = mufu_lg2(rc2);
            v.x = ac.x - (float)kHalfLn2 * fmaf(lgc, f0.x, al.x);
            v.y = ac.y - (float)kHalfLn2 * fmaf(lgc, f0.y, al.y);
          }
        }
        if (S > 1)
          part[buf][unit][qs][lane] = v;
        else
          two_sum(tot, cmp, v);  // points past the column's end add too; they are not stored
      }
      if constexpr (S == 1) {
        // the warp that finishes a stage last fetches the next one into its
        // place; nobody waits for the others
        failed = __any_sync(0xffffffffu, failed);
        if (failed) {  // the copies in flight land before the CTA ends
          tc_mbar_wait(&bar[buf], (kst >> 1) & 1, nullptr, 0);
          if (st + 1 < nstages) tc_mbar_wait(&bar[buf ^ 1], ((kst + 1) >> 1) & 1, nullptr, 0);
          break;
        }
        __syncwarp();  // every lane's reads of the stage, ordered before lane 0's signal
        if (lane == 0) {
          __threadfence_block();
          if (atomicAdd(&done[buf], 1) == WARPS - 1) {
            __threadfence_block();
            done[buf] = 0;
            if (st + 2 < nstages) {
              tc_fence_async_smem();
              fetch(st + 2, buf);
            }
          }
        }
      } else {
        // nobody reads this stage any more and every contribution is in
        failed = __syncthreads_or(failed ? 1 : 0) != 0;
        if (threadIdx.x < kUnits) turn[buf][threadIdx.x] = 0;
        if (sub == 0)
          for (int qs = 0; qs < n; ++qs) two_sum(tot, cmp, part[buf][unit][qs][lane]);
        if (failed) {  // the copies in flight land before the CTA ends
          if (threadIdx.x == 0) {
            tc_mbar_wait(&bar[buf], (kst >> 1) & 1, nullptr, 0);
            if (st + 1 < nstages) tc_mbar_wait(&bar[buf ^ 1], ((kst + 1) >> 1) & 1, nullptr, 0);
          }
          break;
        }
        if (threadIdx.x == 0 && st + 2 < nstages) {
          tc_fence_async_smem();
          fetch(st + 2, buf);
        }
      }
    }
  }
  if (p.work) {
    const unsigned long long npt = live ? min(32, ntp - (i - lane)) : 0;
    terms = __reduce_add_sync(0xffffffffu, terms);
    ndirect = __reduce_add_sync(0xffffffffu, ndirect);
    if (lane == 0 && sub == 0) {
      atomicAdd(&p.work[0], terms * npt);
      atomicAdd(&p.work[1], ndirect * npt);
    }
  }
  if (valid && sub == 0) {
    const double scale = 1.0 / (4.0 * VES_PI);
    double* o = p.out[g] + (long long)col * 2 * ntp;
    o[i] = ((double)tot.x + (double)cmp.x) * scale;
    o[ntp + i] = ((double)tot.y + (double)cmp.y) * scale;
  }
}

// Warps per unit: one from nine units per SM on, four from two per SM, eight
// below.  Measured (one sum, us; S = 1 / 4 / 8): 100 x N=32 (100 units) 195 /
// 45 / 35, 61 x N=128 (244) 276 / 120 / 118, 600 x N=32 (600) 355 / 163 / 203,
// 300 x N=128 (1200) 648 / 592 / 835, 1024 x N=128 (4096) 2050 / 2770 / 3990.
int mp_launch(MPGroupArgs& a, cudaStream_t s) {
  long long units = 0;
  for (int g = 0; g < a.ng; ++g) {
    a.upc[g] = (a.ntp[g] + 31) / 32;
    units += (long long)a.nt[g] * a.upc[g];
  }
  const int S = units >= 152 * 9 ? 1 : units >= 152 * 2 ? 4 : 8;
  const int per = S == 1 ? 4 : 1;  // units per CTA
  a.cta0[0] = 0;
  for (int g = 0; g < a.ng; ++g) a.cta0[g + 1] = a.cta0[g] + (int)(((long long)a.nt[g] * a.upc[g] + per - 1) / per);
  const int grid = a.cta0[a.ng];
  if (grid == 0) return VES_OK;
  ves_count_launch();
  if (S == 1)
    mp_eval_kernel<4, 1><<<grid, 128, 0, s>>>(a);
  else if (S == 4)
    mp_eval_kernel<4, 4><<<grid, 128, 0, s>>>(a);
  else
    mp_eval_kernel<8, 8><<<grid, 256, 0, s>>>(a);
  return ves_launch_check("farfield multipole");
}

}  // namespace

int farfield_mp_run(const FFEnv& env, int nsrc, int ns, const double* Xsrc, const double* den, int nt, int ntp,
                    const double* Xtar, const int* self_idx, const ves_near_lists* nl, double* out, WsCarver& ws,
                    cudaStream_t s) {
  const long long total_pts = (long long)nt * ntp;
  float4* rec = ws.take<float4>((size_t)nsrc * ns);
  MPSrc* src = ws.take<MPSrc>(nsrc);
  MPMom* mom = ws.take<MPMom>((size_t)nsrc * (kPMax + 1));
  float2* tloc = ws.take<float2>((size_t)total_pts);
  float2* thi = ws.take<float2>(nt);
  float2* tlo = ws.take<float2>(nt);
  if (ws.sizing) return VES_OK;
  if (!ws.ok()) {
    ves_record_error(VES_ERR_WORKSPACE, "farfield: workspace too small");
    return VES_ERR_WORKSPACE;
  }
  if (total_pts == 0) return VES_OK;
  if (nsrc == 0) return ves_cuda_status(cudaMemsetAsync(out, 0, (size_t)total_pts * 2 * sizeof(double), s), "ff zero");
  if (ntp > 128) {
    ves_record_error(VES_ERR_SHAPE, "farfield: the multipole path takes at most 128 points per target column");
    return VES_ERR_SHAPE;
  }
  if (nl && ntp != env.N) {
    ves_record_error(VES_ERR_SHAPE, "farfield: near lists need N target points per column");
    return VES_ERR_SHAPE;
  }
  ves_count_launch(2);
  mp_prep_kernel<<<nsrc, 256, 0, s>>>(ns, Xsrc, den, rec, src, mom);
  mp_prep_targets_kernel<<<nt, 256, 0, s>>>(ntp, Xtar, tloc, thi, tlo);
  MPGroupArgs a;
  memset(&a, 0, sizeof(a));
  a.ng = 1;
  a.set[0] = MPSet{nsrc, ns, rec, src, mom};
  a.nt[0] = nt;
  a.ntp[0] = ntp;
  a.tloc[0] = tloc;
  a.thi[0] = thi;
  a.tlo[0] = tlo;
  a.out[0] = out;
  a.self_idx[0] = self_idx;
  a.cand_count[0][0] = nl ? nl->cand_count : nullptr;
  a.cand_src[0][0] = nl ? nl->cand_src : nullptr;
  a.excl_mask[0][0] = nl ? nl->excl_mask : nullptr;
  a.maxc[0][0] = nl ? nl->maxc : 0;
  a.nwords[0] = (env.N + 31) / 32;
  a.work = (env.timing && env.timing->timing) ? env.timing->d_mp : nullptr;
  a.st = env.status;
  if (env.timing) ves_ff_timing_begin(env.timing, s);
  const int rc = mp_launch(a, s);
  if (env.timing) ves_ff_timing_end(env.timing, s, (double)total_pts * ns * (double)nsrc);
  return rc;
}

int farfield_mp_groups_run(const FFEnv& env, int ng, const int* nsrc, const int* ns, const double* const* Xsrc,
                           const double* const* den, const int* nt, const int* ntp, const double* const* Xtar,
                           const ves_near_lists* const* nl, double* const* out, WsCarver& ws, cudaStream_t s) {
  if (ng < 1 || ng > kMPSets) {
    if (!ws.sizing) ves_record_error(VES_ERR_ARG, "farfield groups: 1 to %d point sets", kMPSets);
    return VES_ERR_ARG;
  }
  float4* rec[kMPSets];
  MPSrc* src[kMPSets];
  MPMom* mom[kMPSets];
  float2* tloc[kMPSets];
  long long cols = 0;
  int ntpmax = 0;
  for (int g = 0; g < ng; ++g) {
    rec[g] = ws.take<float4>((size_t)nsrc[g] * ns[g]);
    src[g] = ws.take<MPSrc>(nsrc[g]);
    mom[g] = ws.take<MPMom>((size_t)nsrc[g] * (kPMax + 1));
    tloc[g] = ws.take<float2>((size_t)nt[g] * ntp[g]);
    cols += nt[g];
    ntpmax = std::max(ntpmax, ntp[g]);
  }
  float2* thi = ws.take<float2>((size_t)cols);
  float2* tlo = ws.take<float2>((size_t)cols);
  if (ws.sizing) return VES_OK;
  if (!ws.ok()) {
    ves_record_error(VES_ERR_WORKSPACE, "farfield groups: workspace too small");
    return VES_ERR_WORKSPACE;
  }
  if (cols == 0) return VES_OK;
  if (ntpmax > 128) {
    ves_record_error(VES_ERR_SHAPE, "farfield groups: at most 128 target points per vesicle");
    return VES_ERR_SHAPE;
  }
  MPGroupArgs a;
  memset(&a, 0, sizeof(a));
  a.ng = ng;
  a.st = env.status;
  int col0 = 0;
  for (int g = 0; g < ng; ++g) {
    if (nsrc[g] > 0) {
      ves_count_launch();
      mp_prep_kernel<<<nsrc[g], 256, 0, s>>>(ns[g], Xsrc[g], den[g], rec[g], src[g], mom[g]);
    }
    if (nt[g] > 0) {
      ves_count_launch();
      mp_prep_targets_kernel<<<nt[g], 256, 0, s>>>(ntp[g], Xtar[g], tloc[g], thi + col0, tlo + col0);
    }
    a.set[g] = MPSet{nsrc[g], ns[g], rec[g], src[g], mom[g]};
    a.nt[g] = nt[g];
    a.ntp[g] = ntp[g];
    a.tloc[g] = tloc[g];
    a.thi[g] = thi + col0;
    a.tlo[g] = tlo + col0;
    a.out[g] = out[g];
    a.own[g] = 1;
    col0 += nt[g];
    a.nwords[g] = (ntp[g] + 31) / 32;
    for (int q = 0; q < ng; ++q) {
      const ves_near_lists* L = nl ? nl[g * ng + q] : nullptr;
      a.cand_count[g][q] = L ? L->cand_count : nullptr;
      a.cand_src[g][q] = L ? L->cand_src : nullptr;
      a.excl_mask[g][q] = L ? L->excl_mask : nullptr;
      a.maxc[g][q] = L ? L->maxc : 0;
    }
  }
  return mp_launch(a, s);
}
