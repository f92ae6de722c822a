// Near-zone lists built on the device and the near-singular corrections.
//
// Candidate search: every target vesicle scans all vesicles with one warp,
// testing bounding boxes grown by the near threshold; hits are appended in
// ascending order (warp ballot + popc), so each target vesicle owns a sorted
// candidate list ("bucket") that the far-field kernel walks with a cursor.
// Point-level tests then run one CTA per (target vesicle, candidate).
//
// Two schemes:
// * py_hh — naiveNearZoneInfo (mytorch/biem_support.py:520-613) and
//   nearSingInt_hh (mytorch/poten.py:466-600).  Exclusions: target point i of t
//   is near source vesicle s if any of the Nup upsampled points of s lies
//   closer than the threshold.  Correction: the reference's hedgehog list is
//   indexed by (t, s*Nup + u) but consumed as if it were (k1, k2*N + J); for
//   every such entry with k2 != k1 it adds vself[(icp - 3) mod N, k1] at
//   (J, k2), where icp is the coarse point of k1 closest to upsampled point J
//   of k2 (the last row of the Lagrange matrix is e_0, poten.py:987, so the
//   interpolated value is the first stencil value).
// * matlab — getZone/closestPnt (matlab/capsules_py.m:194-643) and nearSingInt
//   (matlab/poten_py.m:495-692): near if the Newton closest point on the local
//   7-point interpolant of s is closer than h; the trapezoid contribution of s
//   is removed (exclusion) and replaced by the 7-point Lagrange extrapolation
//   along the normal, evaluated at dist/(6*beta*h).
#include "ves_internal.h"

namespace {

__device__ __forceinline__ double horner7(const double* c, double t) {
  double v = 0.0;
#pragma unroll
  for (int i = 0; i < 7; ++i) v = fma(v, t, c[i]);
  return v;
}

// bounding boxes [nv][4] = xmin, xmax, ymin, ymax of n-point curves.  A
// curve with a non-finite coordinate gets the empty box (+inf, -inf, +inf,
// -inf), which meets no other box, and raises VES_ERR_NONFINITE (site 22,
// detail = the vesicle): a NaN must not turn into a near pair with every
// vesicle.
__global__ void bbox_kernel(int n, const double* __restrict__ X, double* __restrict__ box,
                            VesDeviceStatus* st) {
  __shared__ double red[4][128];
  __shared__ int bad;
  const int k = blockIdx.x;
  const double* x = X + (long long)k * 2 * n;
  if (threadIdx.x == 0) bad = 0;
  __syncthreads();
  double a = 1e300, b = -1e300, c = 1e300, d = -1e300;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    const double xv = x[j], yv = x[n + j];
    if (!isfinite(xv) || !isfinite(yv)) bad = 1;
    a = fmin(a, xv);
    b = fmax(b, xv);
    c = fmin(c, yv);
    d = fmax(d, yv);
  }
  red[0][threadIdx.x] = a;
  red[1][threadIdx.x] = b;
  red[2][threadIdx.x] = c;
  red[3][threadIdx.x] = d;
  __syncthreads();
  for (int w = 64; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      red[0][threadIdx.x] = fmin(red[0][threadIdx.x], red[0][threadIdx.x + w]);
      red[1][threadIdx.x] = fmax(red[1][threadIdx.x], red[1][threadIdx.x + w]);
      red[2][threadIdx.x] = fmin(red[2][threadIdx.x], red[2][threadIdx.x + w]);
      red[3][threadIdx.x] = fmax(red[3][threadIdx.x], red[3][threadIdx.x + w]);
    }
    __syncthreads();
  }
  if (threadIdx.x < 4) {
    const double inf = __longlong_as_double(0x7ff0000000000000LL);
    box[k * 4 + threadIdx.x] = bad ? ((threadIdx.x & 1) ? -inf : inf) : red[threadIdx.x][0];
  }
  if (threadIdx.x == 0 && bad) ves_set_error(st, VES_ERR_NONFINITE, 22, (long long)k);
}

// ---- bucket-sorted candidate search ----------------------------------------
// The source boxes' centres are counting-sorted into a uniform grid whose
// cell is at least (max target box + max source box)/2 + threshold wide, so
// every source whose box comes within the threshold of a target's box has
// its centre in one of the 3 x 3 cells around the target's centre.  One warp
// per target then tests the boxes of those cells only: O(nv) work for a
// suspension instead of O(nv^2).
struct GridParams {
  double x0, y0, inv_cell;
  int nx, ny;
};

__device__ __forceinline__ bool box_valid(const double* b) { return b[0] <= b[1] && b[2] <= b[3]; }

// one block of 1024 threads: extents of the valid boxes, cell size and grid
// dimensions (at most cap_cells cells)
__global__ void __launch_bounds__(1024) grid_setup_kernel(int ns, const double* __restrict__ sbox, int nt,
                                                          const double* __restrict__ tbox, double thr, int cap_cells,
                                                          GridParams* __restrict__ gp) {
  double x0 = 1e300, x1 = -1e300, y0 = 1e300, y1 = -1e300, ws = 0.0, wt = 0.0;
  for (int i = threadIdx.x; i < ns; i += blockDim.x) {
    const double* b = sbox + 4 * (long long)i;
    if (!box_valid(b)) continue;
    const double cx = 0.5 * (b[0] + b[1]), cy = 0.5 * (b[2] + b[3]);
    x0 = fmin(x0, cx);
    x1 = fmax(x1, cx);
    y0 = fmin(y0, cy);
    y1 = fmax(y1, cy);
    ws = fmax(ws, fmax(b[1] - b[0], b[3] - b[2]));
  }
  for (int i = threadIdx.x; i < nt; i += blockDim.x) {
    const double* b = tbox + 4 * (long long)i;
    if (box_valid(b)) wt = fmax(wt, fmax(b[1] - b[0], b[3] - b[2]));
  }
  // reduce: min x0,y0 (as -max of negatives), max x1,y1,ws,wt
  double v[6] = {-x0, x1, -y0, y1, ws, wt};
  for (int q = 0; q < 6; ++q)
    for (int o = 16; o > 0; o >>= 1) v[q] = fmax(v[q], __shfl_xor_sync(0xffffffffu, v[q], o));
  __shared__ double part[6][32];
  const int w = threadIdx.x / 32, l = threadIdx.x % 32;
  if (l == 0)
    for (int q = 0; q < 6; ++q) part[q][w] = v[q];
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x / 32;
    for (int q = 0; q < 6; ++q) {
      double t = l < nw ? part[q][l] : -1e300;
      for (int o = 16; o > 0; o >>= 1) t = fmax(t, __shfl_xor_sync(0xffffffffu, t, o));
      v[q] = t;
    }
    if (l == 0) {
      GridParams g;
      double gx0 = -v[0], gx1 = v[1], gy0 = -v[2], gy1 = v[3];
      if (!(gx0 <= gx1)) gx0 = gx1 = gy0 = gy1 = 0.0;  // no valid source box
      double cell = 0.5 * (v[4] + fmax(v[5], 0.0)) + thr;
      if (!(cell > 0.0)) cell = 1.0;
      const double ex = gx1 - gx0, ey = gy1 - gy0;
      // grow the cell until the grid has at most cap_cells cells
      for (int it = 0; it < 64; ++it) {
        const double nx = floor(ex / cell) + 1.0, ny = floor(ey / cell) + 1.0;
        if (nx * ny <= (double)cap_cells) break;
        cell *= 1.25;
      }
      g.x0 = gx0;
      g.y0 = gy0;
      g.inv_cell = 1.0 / cell;
      g.nx = (int)(floor(ex / cell) + 1.0);
      g.ny = (int)(floor(ey / cell) + 1.0);
      if (g.nx < 1) g.nx = 1;
      if (g.ny < 1) g.ny = 1;
      if ((long long)g.nx * g.ny > cap_cells) g.nx = g.ny = 1;  // unreachable for finite extents
      *gp = g;
    }
  }
}

__device__ __forceinline__ int grid_coord(double c, double c0, double inv, int n) {
  const double f = floor((c - c0) * inv);
  return (int)fmin(fmax(f, -2.0), (double)n + 1.0);  // off-grid targets stay off-grid
}

__global__ void grid_count_kernel(int ns, const double* __restrict__ sbox, const GridParams* __restrict__ gp,
                                  int* __restrict__ cell_of, int* __restrict__ counts) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ns) return;
  const double* b = sbox + 4 * (long long)i;
  if (!box_valid(b)) {
    cell_of[i] = -1;
    return;
  }
  const GridParams g = *gp;
  const int cx = min(max(grid_coord(0.5 * (b[0] + b[1]), g.x0, g.inv_cell, g.nx), 0), g.nx - 1);
  const int cy = min(max(grid_coord(0.5 * (b[2] + b[3]), g.y0, g.inv_cell, g.ny), 0), g.ny - 1);
  const int cell = cy * g.nx + cx;
  cell_of[i] = cell;
  atomicAdd(&counts[cell], 1);
}

// exclusive scan of n counts (one block of 1024 threads); start[n] = total
__global__ void __launch_bounds__(1024) scan_kernel(int n, const int* __restrict__ counts, int* __restrict__ start) {
  __shared__ int wsum[32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x % 32, w = threadIdx.x / 32;
  for (int base = 0; base < n; base += blockDim.x) {
    const int i = base + threadIdx.x;
    const int v = i < n ? counts[i] : 0;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
      int t = wsum[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += y;
      }
      wsum[lane] = t;
    }
    __syncthreads();
    const int excl = carry + (w > 0 ? wsum[w - 1] : 0) + x - v;
    if (i < n) start[i] = excl;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = excl + v;
    __syncthreads();
  }
  if (threadIdx.x == 0) start[n] = carry;
}

__global__ void grid_fill_kernel(int ns, const int* __restrict__ cell_of, const int* __restrict__ start,
                                 int* __restrict__ fill, int* __restrict__ sorted) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ns || cell_of[i] < 0) return;
  const int c = cell_of[i];
  sorted[start[c] + atomicAdd(&fill[c], 1)] = i;
}

// one warp per target vesicle: boxes of the 3 x 3 cells around its centre;
// hits appended (order fixed by sort_candidates_kernel); the true count is
// kept for the capacity check
__global__ void grid_candidates_kernel(int nt, bool same_set, const double* __restrict__ tbox,
                                       const double* __restrict__ sbox, double thr, const GridParams* __restrict__ gp,
                                       const int* __restrict__ start, const int* __restrict__ sorted, int maxc,
                                       int* __restrict__ cand_count, int* __restrict__ cand_src,
                                       int* __restrict__ max_count) {
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
  const int lane = threadIdx.x % 32;
  if (t >= nt) return;
  const double* tb = tbox + 4 * (long long)t;
  int count = 0;
  if (box_valid(tb)) {
    const GridParams g = *gp;
    const double tx0 = tb[0], tx1 = tb[1], ty0 = tb[2], ty1 = tb[3];
    const int ix = grid_coord(0.5 * (tx0 + tx1), g.x0, g.inv_cell, g.nx);
    const int iy = grid_coord(0.5 * (ty0 + ty1), g.y0, g.inv_cell, g.ny);
    for (int cy = max(iy - 1, 0); cy <= min(iy + 1, g.ny - 1); ++cy)
      for (int cx = max(ix - 1, 0); cx <= min(ix + 1, g.nx - 1); ++cx) {
        const int cell = cy * g.nx + cx;
        const int b0 = start[cell], b1 = start[cell + 1];
        for (int base = b0; base < b1; base += 32) {
          const int k = base + lane;
          bool hit = false;
          int sidx = -1;
          if (k < b1) {
            sidx = sorted[k];
            if (!(same_set && sidx == t)) {
              const double* sb = sbox + 4 * (long long)sidx;
              const double gx = fmax(0.0, fmax(sb[0] - tx1, tx0 - sb[1]));
              const double gy = fmax(0.0, fmax(sb[2] - ty1, ty0 - sb[3]));
              hit = gx * gx + gy * gy < thr * thr;
            }
          }
          const unsigned m = __ballot_sync(0xffffffffu, hit);
          const int pos = count + __popc(m & ((1u << lane) - 1u));
          if (hit && pos < maxc) cand_src[(long long)t * maxc + pos] = sidx;
          count += __popc(m);
        }
      }
  }
  if (lane == 0) {
    cand_count[t] = count < maxc ? count : maxc;
    atomicMax(max_count, count);
  }
}

// ascending order of each target's candidate list (the far-field kernels
// walk the lists with a cursor); one block per target, rank sort in shared
// memory (the lists hold distinct vesicle indices)
__global__ void sort_candidates_kernel(int maxc, const int* __restrict__ cand_count, int* __restrict__ cand_src) {
  extern __shared__ int lst[];
  const int t = blockIdx.x;
  const int n = cand_count[t];
  if (n <= 1) return;
  int* row = cand_src + (long long)t * maxc;
  for (int i = threadIdx.x; i < n; i += blockDim.x) lst[i] = row[i];
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int v = lst[i];
    int r = 0;
    for (int j = 0; j < n; ++j) r += lst[j] < v;
    row[r] = v;
  }
}

// py scheme: exclusion bits per target point and hedgehog bits per upsampled point
__global__ void __launch_bounds__(256) py_masks_kernel(int N, int Nup, int maxc, double thr2,
                                                       const double* __restrict__ X, const double* __restrict__ Xup,
                                                       const int* __restrict__ cand_count,
                                                       const int* __restrict__ cand_src,
                                                       uint32_t* __restrict__ excl_mask,
                                                       uint32_t* __restrict__ hh_mask) {
  extern __shared__ double sh[];
  const int t = blockIdx.y, slot = blockIdx.x;
  const int wN = (N + 31) / 32, wU = (Nup + 31) / 32;
  uint32_t* em = excl_mask + ((long long)t * maxc + slot) * wN;
  uint32_t* hm = hh_mask + ((long long)t * maxc + slot) * wU;
  if (slot >= cand_count[t]) return;
  const int s = cand_src[(long long)t * maxc + slot];
  double* tx = sh;
  double* ty = tx + N;
  uint32_t* ebits = (uint32_t*)(ty + N);
  uint32_t* hbits = ebits + wN;
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    tx[i] = X[(long long)t * 2 * N + i];
    ty[i] = X[(long long)t * 2 * N + N + i];
  }
  for (int i = threadIdx.x; i < wN; i += blockDim.x) ebits[i] = 0;
  for (int i = threadIdx.x; i < wU; i += blockDim.x) hbits[i] = 0;
  __syncthreads();
  const double* xs = Xup + (long long)s * 2 * Nup;
  for (int u = threadIdx.x; u < Nup; u += blockDim.x) {
    const double sx = xs[u], sy = xs[Nup + u];
    bool any = false;
    for (int i = 0; i < N; ++i) {
      const double dx = tx[i] - sx, dy = ty[i] - sy;
      if (dx * dx + dy * dy < thr2) {
        any = true;
        atomicOr(&ebits[i >> 5], 1u << (i & 31));
      }
    }
    if (any) atomicOr(&hbits[u >> 5], 1u << (u & 31));
  }
  __syncthreads();
  for (int i = threadIdx.x; i < wN; i += blockDim.x) em[i] = ebits[i];
  for (int i = threadIdx.x; i < wU; i += blockDim.x) hm[i] = hbits[i];
}

// py_hh correction.  Bit u of a pair (t, s) of the lists is the hedgehog point
// of upsampled point u of s: read as (k2, J) with s Nup + u = k2 N + J it adds
// the self velocity of t at the coarse point of t three before the closest one
// to upsampled point J of k2.
__device__ __forceinline__ bool hh_point(int nv, int N, int Nup, int t, int s, int u, int& k2, int& J) {
  const int q = u / N;  // Nup is a multiple of N
  k2 = s * (Nup / N) + q;
  J = u - q * N;
  return k2 < nv && k2 != t;
}

// The vesicles t that add to a point: hits[0][nv][N] counts them (zero before the
// launch), hits[1..kHits][nv][N] has up to kHits of them in any order.
constexpr int kHits = VES_HEDGEHOG_HITS - 1;
__global__ void __launch_bounds__(128) hh_count_kernel(int nv, int N, int Nup, int maxc,
                                                       const int* __restrict__ cand_count,
                                                       const int* __restrict__ cand_src,
                                                       const uint32_t* __restrict__ hh_mask, int* __restrict__ hits) {
  const int t = blockIdx.x, wU = (Nup + 31) / 32;
  const int nc = min(cand_count[t], maxc);
  const size_t n = (size_t)nv * N;
  for (int i = threadIdx.x; i < nc * wU; i += blockDim.x) {
    const int slot = i / wU, w = i - slot * wU;
    uint32_t bits = hh_mask[((long long)t * maxc + slot) * wU + w];
    if (bits == 0u) continue;
    const int s = cand_src[(long long)t * maxc + slot];
    for (; bits; bits &= bits - 1) {
      int k2, J;
      if (!hh_point(nv, N, Nup, t, s, w * 32 + __ffs(bits) - 1, k2, J)) continue;
      const size_t p = (size_t)k2 * N + J;
      const int at = atomicAdd(&hits[p], 1);
      if (at < kHits) hits[(size_t)(1 + at) * n + p] = t;
    }
  }
}

// The first vesicle from t0 on that adds to the point (u of s, J of k2), nv if
// none: by the lists, for a point of more than kHits.
__device__ __forceinline__ int hh_scan(int nv, int Nup, int maxc, const int* __restrict__ cand_count,
                                       const int* __restrict__ cand_src, const uint32_t* __restrict__ hh_mask, int t0,
                                       int k2, int s, int u, int lane) {
  const int wU = (Nup + 31) / 32;
  for (int b = t0; b < nv; b += 32) {
    const int t = b + lane;
    bool bit = false;
    if (t < nv && t != k2) {
      const int* row = cand_src + (long long)t * maxc;
      const int nc = min(cand_count[t], maxc);
      int lo = 0, hi = nc;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (row[mid] < s) lo = mid + 1; else hi = mid;
      }
      bit = lo < nc && row[lo] == s && ((hh_mask[((long long)t * maxc + lo) * wU + (u >> 5)] >> (u & 31)) & 1u);
    }
    const unsigned m = __ballot_sync(0xffffffffu, bit);
    if (m) return b + __ffs(m) - 1;
  }
  return nv;
}

// One CTA per vesicle t.  Latency-bound: a hedgehog point is a search of the N
// coarse points (FP64 distances), and the points of a close pair sit side by
// side, that is in one or two words of the mask.  So the warps take the set
// bits in turn and the lanes share one point's search (30 us a call at 301
// vesicles of N = 64).  A point that several vesicles add to is taken by the
// warp of the first of them, which adds the others' values after its own in
// ascending order: the sum does not depend on which CTA is first.
__global__ void __launch_bounds__(128) hh_apply_kernel(int nv, int N, int Nup, int maxc, const double* __restrict__ X,
                                                       const double* __restrict__ Xup,
                                                       const int* __restrict__ cand_count,
                                                       const int* __restrict__ cand_src,
                                                       const uint32_t* __restrict__ hh_mask,
                                                       const int* __restrict__ hits,
                                                       const double* __restrict__ vself, double* __restrict__ LP,
                                                       double* __restrict__ near_only) {
  extern __shared__ double xk[];  // [2][N] coarse points of t (k1 of every pair)
  const int t = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int nc = min(cand_count[t], maxc);
  if (nc <= 0) return;
  for (int i = threadIdx.x; i < 2 * N; i += blockDim.x) xk[i] = X[(long long)t * 2 * N + i];
  __syncthreads();
  const int wU = (Nup + 31) / 32;
  const size_t n = (size_t)nv * N;
  // the value of vesicle t1 (coarse points x) at upsampled point J of k2
  auto add = [&](int t1, const double* x, int k2, int J, double px, double py) {
    double best = 1e300;
    int icp = 0x7fffffff;  // closest coarse point (first minimum)
    for (int i = lane; i < N; i += 32) {
      const double dx = x[i] - px, dy = x[N + i] - py;
      const double d2 = dx * dx + dy * dy;
      if (d2 < best) {
        best = d2;
        icp = i;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double d2 = __shfl_xor_sync(0xffffffffu, best, o);
      const int i2 = __shfl_xor_sync(0xffffffffu, icp, o);
      if (d2 < best || (d2 == best && i2 < icp)) {
        best = d2;
        icp = i2;
      }
    }
    if (icp == 0x7fffffff) icp = 0;  // no finite distance
    const int pn0 = ((icp - 3) % N + N) % N;
    if (lane < 2) {  // one component each
      const double v = vself[(long long)t1 * 2 * N + lane * N + pn0];
      atomicAdd(&LP[(long long)k2 * 2 * N + lane * N + J], v);
      if (near_only) atomicAdd(&near_only[(long long)k2 * 2 * N + lane * N + J], v);
    }
  };
  int turn = 0;  // set bits so far: each belongs to one warp
  for (int slot = 0; slot < nc; ++slot) {
    const int s = cand_src[(long long)t * maxc + slot];
    const uint32_t* hm = hh_mask + ((long long)t * maxc + slot) * wU;
    for (int w0 = 0; w0 < wU; w0 += 32) {
      const uint32_t word = w0 + lane < wU ? hm[w0 + lane] : 0u;
      unsigned some = __ballot_sync(0xffffffffu, word != 0u);
      while (some) {
        const int wl = __ffs(some) - 1;
        some &= some - 1;
        uint32_t bits = __shfl_sync(0xffffffffu, word, wl);
        while (bits) {
          const int b = __ffs(bits) - 1;
          bits &= bits - 1;
          if (turn++ % nw != warp) continue;
          const int u = (w0 + wl) * 32 + b;
          int k2, J;
          if (!hh_point(nv, N, Nup, t, s, u, k2, J)) continue;
          const size_t p = (size_t)k2 * N + J;
          const int m = hits[p];
          const double px = Xup[(long long)k2 * 2 * Nup + J], py = Xup[(long long)k2 * 2 * Nup + Nup + J];
          if (m <= 1) {
            add(t, xk, k2, J, px, py);
            continue;
          }
          const int own = m <= kHits && lane < m ? hits[(size_t)(1 + lane) * n + p] : nv;  // a vesicle per lane
          auto next = [&](int t0) {  // the first of them from t0 on
            return m <= kHits ? (int)__reduce_min_sync(0xffffffffu, (unsigned)(own >= t0 ? own : nv))
                              : hh_scan(nv, Nup, maxc, cand_count, cand_src, hh_mask, t0, k2, s, u, lane);
          };
          if (next(0) != t) continue;
          for (int t1 = t; t1 < nv; t1 = next(t1 + 1)) add(t1, X + (long long)t1 * 2 * N, k2, J, px, py);
        }
      }
    }
  }
}

// MATLAB scheme: per (target vesicle t, candidate source s) and target point j;
// targets Xt with Nt points per vesicle, sources Xs with Ns (one set: Xt = Xs)
__global__ void __launch_bounds__(128) matlab_zone_kernel(int Nt, int Ns, int maxc, double h,
                                                          const double* __restrict__ Xt,
                                                          const double* __restrict__ Xs,
                                                          const double* __restrict__ lag,
                                                          const int* __restrict__ cand_count,
                                                          const int* __restrict__ cand_src,
                                                          uint32_t* __restrict__ excl_mask, int max_entries,
                                                          int* __restrict__ n_entries, int* __restrict__ ent_tsj,
                                                          int* __restrict__ ent_icp, double* __restrict__ ent_geo,
                                                          VesDeviceStatus* st) {
  extern __shared__ double sh[];
  const int t = blockIdx.y, slot = blockIdx.x;
  const int wN = (Nt + 31) / 32;
  uint32_t* em = excl_mask + ((long long)t * maxc + slot) * wN;
  if (slot >= cand_count[t]) return;
  const int s = cand_src[(long long)t * maxc + slot];
  double* sx = sh;
  double* sy = sx + Ns;
  double* L = sy + Ns;  // 49
  uint32_t* bits = (uint32_t*)(L + 49);
  for (int i = threadIdx.x; i < Ns; i += blockDim.x) {
    sx[i] = Xs[(long long)s * 2 * Ns + i];
    sy[i] = Xs[(long long)s * 2 * Ns + Ns + i];
  }
  for (int i = threadIdx.x; i < 49; i += blockDim.x) L[i] = lag[i];
  for (int i = threadIdx.x; i < wN; i += blockDim.x) bits[i] = 0;
  __syncthreads();
  for (int j = threadIdx.x; j < Nt; j += blockDim.x) {
    const double xt = Xt[(long long)t * 2 * Nt + j], yt = Xt[(long long)t * 2 * Nt + Nt + j];
    double best = 1e300;
    int icp = 0;
    for (int i = 0; i < Ns; ++i) {
      const double dx = xt - sx[i], dy = yt - sy[i];
      const double d2 = dx * dx + dy * dy;
      if (d2 < best) {
        best = d2;
        icp = i;
      }
    }
    if (sqrt(best) >= 2.0 * h) continue;
    // closestPnt: one Newton step from theta = 1/2 on the 7-point interpolant
    double px[7], py[7];
#pragma unroll
    for (int r = 0; r < 7; ++r) {
      double ax = 0, ay = 0;
#pragma unroll
      for (int q = 0; q < 7; ++q) {
        const int idx = ((icp - 3 + q) % Ns + Ns) % Ns;
        ax = fma(L[r * 7 + q], sx[idx], ax);
        ay = fma(L[r * 7 + q], sy[idx], ay);
      }
      px[r] = ax;
      py[r] = ay;
    }
    double dpx[6], dpy[6], d2px[5], d2py[5];
#pragma unroll
    for (int r = 0; r < 6; ++r) {
      dpx[r] = px[r] * (6 - r);
      dpy[r] = py[r] * (6 - r);
    }
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      d2px[r] = dpx[r] * (5 - r);
      d2py[r] = dpy[r] * (5 - r);
    }
    auto hp = [](const double* c, int n, double x) {
      double v = 0;
      for (int i = 0; i < n; ++i) v = fma(v, x, c[i]);
      return v;
    };
    double th = 0.5;
    const double zx = hp(px, 7, th), zy = hp(py, 7, th);
    const double dzx = hp(dpx, 6, th), dzy = hp(dpy, 6, th);
    const double d2zx = hp(d2px, 5, th), d2zy = hp(d2py, 5, th);
    const double num = (zx - xt) * dzx + (zy - yt) * dzy;
    const double den = (zx - xt) * d2zx + (zy - yt) * d2zy + dzx * dzx + dzy * dzy;
    th = th - num / den;
    const double nx = hp(px, 7, th), ny = hp(py, 7, th);
    const double dist = sqrt((nx - xt) * (nx - xt) + (ny - yt) * (ny - yt));
    if (dist < h) {
      atomicOr(&bits[j >> 5], 1u << (j & 31));
      const int e = atomicAdd(n_entries, 1);
      if (e < max_entries) {
        ent_tsj[3 * e] = t;
        ent_tsj[3 * e + 1] = s;
        ent_tsj[3 * e + 2] = j;
        ent_icp[e] = icp;
        ent_geo[4 * e] = dist;
        ent_geo[4 * e + 1] = nx;
        ent_geo[4 * e + 2] = ny;
        ent_geo[4 * e + 3] = th;
      } else {
        ves_set_error(st, VES_ERR_NEARLIST_OVERFLOW, 21, e);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < wN; i += blockDim.x) em[i] = bits[i];
}

// MATLAB correction.  DL: the layer potential at the Lagrange points is the
// double layer (kernelDirect = exactStokesDL, tstep_biem.py:236,501), with
// normals (ty, -tx) of the upsampled source and den already scaled by
// (1 - visc); otherwise the single layer.
// One correction problem: targets of a point set (Xt and LP, Nt points per
// vesicle) against the sources (vself with Ns points; Xup, tang_up and den
// with Nup upsampled points) of another set or of itself, with the near
// entries of its lists.
struct MatlabPair {
  int set;  // number of the target set: problems of one set add to the same LP
  int nvt, Nt, Ns, Nup;
  double h;
  const double *Xt, *Xup, *tang_up, *den, *vself, *lag;
  const int* n_entries;
  int max_entries, maxc;
  const int *ent_tsj, *ent_icp;
  const double* ent_geo;
  const int* cand_count;
  const uint32_t* excl_mask;
  double *LP, *near_only;
};

// Several correction problems (every pair of point sets of a suspension with
// several point counts) in one launch: problem k owns the warps
// [warp0[k], warp0[k+1]), one per near-entry slot.  The index (or null) chains
// the slots of each target point: head[k][t Nt + j] is one of them and next[w]
// the one after slot w, -1 at the end; problems of one target set share their
// chains.
constexpr int kMatlabPairs = 16;
struct MatlabPairs {
  int np;
  long long warp0[kMatlabPairs + 1];
  MatlabPair pair[kMatlabPairs];
  int* next;
  int* head[kMatlabPairs];
};

__device__ __forceinline__ int matlab_problem(const MatlabPairs& P, long long w) {
  int k = 0;
  while (k + 1 < P.np && w >= P.warp0[k + 1]) ++k;
  return k;
}

// one thread per slot (heads are -1 before the launch)
__global__ void __launch_bounds__(256) matlab_index_kernel(const __grid_constant__ MatlabPairs P) {
  const long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= P.warp0[P.np]) return;
  const int k = matlab_problem(P, w), e = (int)(w - P.warp0[k]);
  const MatlabPair& a = P.pair[k];
  if (e >= min(*a.n_entries, a.max_entries)) return;
  const long long at = (long long)a.ent_tsj[3 * (long long)e] * a.Nt + a.ent_tsj[3 * (long long)e + 2];
  P.next[w] = atomicExch(&P.head[k][at], (int)w);
}

// Problem, source vesicle and list place of an entry, in the order in which
// the entries of one target point are added.
typedef unsigned long long MatlabKey;
static_assert(kMatlabPairs <= 16, "four bits of a key");
constexpr MatlabKey kNoEntry = ~0ull;
__device__ __forceinline__ MatlabKey matlab_key(int k, int s, int e) {
  return ((MatlabKey)k << 60) | ((MatlabKey)(unsigned)s << 32) | (unsigned)e;
}

// true if point j of target vesicle t lies near more than one source vesicle
// of the problems that add to problem k0's points: by its chain, or by the
// lists' masks (the warp's lanes share the slots)
__device__ __forceinline__ bool matlab_shared(const MatlabPairs& P, int k0, int t, int j, int lane) {
  if (P.next) return P.next[P.head[k0][(long long)t * P.pair[k0].Nt + j]] >= 0;
  const int set = P.pair[k0].set;
  int n = 0;
  for (int k = 0; k < P.np; ++k) {
    const MatlabPair& a = P.pair[k];
    if (a.set != set || !a.cand_count || !a.excl_mask) continue;
    const int cc = min(a.cand_count[t], a.maxc), nw = (a.Nt + 31) / 32;
    const uint32_t* m = a.excl_mask + (long long)t * a.maxc * nw + (j >> 5);
    for (int s0 = 0; s0 < cc; s0 += 32) {
      const bool bit = s0 + lane < cc && ((m[(long long)(s0 + lane) * nw] >> (j & 31)) & 1u);
      n += __popc(__ballot_sync(0xffffffffu, bit));
    }
  }
  return n > 1;
}

// the first entry of point (t, j) of problem k's targets at or after key `from`
// (kNoEntry: none): along the point's chain, or without one in all lists
__device__ __forceinline__ MatlabKey matlab_next(const MatlabPairs& P, int k0, int t, int j, MatlabKey from, int lane) {
  MatlabKey best = kNoEntry;
  if (P.next) {
    for (int w = P.head[k0][(long long)t * P.pair[k0].Nt + j]; w >= 0; w = P.next[w]) {
      const int k = matlab_problem(P, w), e = (int)(w - P.warp0[k]);
      const MatlabKey key = matlab_key(k, P.pair[k].ent_tsj[3 * (long long)e + 1], e);
      if (key >= from && key < best) best = key;
    }
    return best;
  }
  const int set = P.pair[k0].set;
  for (int k = 0; k < P.np; ++k) {
    const MatlabPair& a = P.pair[k];
    if (a.set != set) continue;
    const int ne = min(*a.n_entries, a.max_entries);
#pragma unroll 4
    for (int e = lane; e < ne; e += 32) {
      if (a.ent_tsj[3 * e] != t || a.ent_tsj[3 * e + 2] != j) continue;
      const MatlabKey key = matlab_key(k, a.ent_tsj[3 * e + 1], e);
      if (key >= from && key < best) best = key;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const MatlabKey b = __shfl_xor_sync(0xffffffffu, best, o);
    if (b < best) best = b;
  }
  return best;
}

// Near entry e of problem a (target t, source s, point j), one warp: its value
// is added to LP by lane 0.
template <bool DL>
__device__ __forceinline__ void matlab_add_entry(const MatlabPair& a, int e, int lane) {
  const int t = a.ent_tsj[3 * e], s = a.ent_tsj[3 * e + 1], j = a.ent_tsj[3 * e + 2];
  const int icp = a.ent_icp[e];
  const double dist = a.ent_geo[4 * e], nxp = a.ent_geo[4 * e + 1], nyp = a.ent_geo[4 * e + 2], th = a.ent_geo[4 * e + 3];
  const double beta = 1.1;
  const double xt = a.Xt[(long long)t * 2 * a.Nt + j], yt = a.Xt[(long long)t * 2 * a.Nt + a.Nt + j];
  const double ux = (xt - nxp) / dist, uy = (yt - nyp) / dist;
  // layer potential of source vesicle s at the 6 Lagrange points
  double ax[6], ay[6];
#pragma unroll
  for (int m = 0; m < 6; ++m) ax[m] = ay[m] = 0.0;
  const double* xs = a.Xup + (long long)s * 2 * a.Nup;
  const double* ds = a.den + (long long)s * 2 * a.Nup;
  for (int u = lane; u < a.Nup; u += 32) {
    const double sxu = xs[u], syu = xs[a.Nup + u], dxu = ds[u], dyu = ds[a.Nup + u];
    double nxu = 0.0, nyu = 0.0;
    if (DL) {
      nxu = a.tang_up[(long long)s * 2 * a.Nup + a.Nup + u];
      nyu = -a.tang_up[(long long)s * 2 * a.Nup + u];
    }
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const double px = nxp + beta * a.h * ux * (m + 1), py = nyp + beta * a.h * uy * (m + 1);
      const double rx = px - sxu, ry = py - syu;
      const double r2 = rx * rx + ry * ry;
      if (DL) {
        const double cc = ((rx * nxu + ry * nyu) / (r2 * r2)) * (rx * dxu + ry * dyu);
        ax[m] += cc * rx;
        ay[m] += cc * ry;
      } else {
        const double lg = 0.5 * log(r2);
        const double cc = (rx * dxu + ry * dyu) / r2;
        ax[m] += cc * rx - lg * dxu;
        ay[m] += cc * ry - lg * dyu;
      }
    }
  }
#pragma unroll
  for (int m = 0; m < 6; ++m) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ax[m] += __shfl_xor_sync(0xffffffffu, ax[m], o);
      ay[m] += __shfl_xor_sync(0xffffffffu, ay[m], o);
    }
  }
  if (lane != 0) return;
  const double kscale = DL ? 1.0 / VES_PI : 1.0 / (4.0 * VES_PI);
  double vals[2];
  for (int comp = 0; comp < 2; ++comp) {
    // on-curve value: Lagrange interpolant of vself around icp at theta
    double coef[7], stencil[7];
    for (int q = 0; q < 7; ++q) stencil[q] = a.vself[(long long)s * 2 * a.Ns + comp * a.Ns + ((icp - 3 + q) % a.Ns + a.Ns) % a.Ns];
    for (int r = 0; r < 7; ++r) {
      double acc = 0;
      for (int q = 0; q < 7; ++q) acc = fma(a.lag[r * 7 + q], stencil[q], acc);
      coef[r] = acc;
    }
    const double vel = horner7(coef, th);
    double pts[7];
    pts[0] = vel;
    for (int m = 0; m < 6; ++m) pts[m + 1] = (comp == 0 ? ax[m] : ay[m]) * kscale;
    for (int r = 0; r < 7; ++r) {
      double acc = 0;
      for (int q = 0; q < 7; ++q) acc = fma(a.lag[r * 7 + q], pts[q], acc);
      coef[r] = acc;
    }
    vals[comp] = horner7(coef, dist / (beta * a.h * 6.0));
  }
  atomicAdd(&a.LP[(long long)t * 2 * a.Nt + j], vals[0]);
  atomicAdd(&a.LP[(long long)t * 2 * a.Nt + a.Nt + j], vals[1]);
  if (a.near_only) {
    atomicAdd(&a.near_only[(long long)t * 2 * a.Nt + j], vals[0]);
    atomicAdd(&a.near_only[(long long)t * 2 * a.Nt + a.Nt + j], vals[1]);
  }
}

// One warp per near entry.  A point near one source takes one addition.  The
// entries of a point near several sources (of one set or of several) are all
// added by the warp of the first of them, in ascending order of (problem,
// source), so that the sum does not depend on the order of the lists or of the
// warps.  FP64 arithmetic (six layer potentials over Nup points per entry)
// bounds the kernel.  CTAs of two warps: a warp with two or three entries holds
// no others' places (with eight warps to a CTA 8192 x N=32, 50617 entries, 7.1
// ms, with two 6.6), and few entries spread over the chip (1024 x N=128 1.06 ->
// 0.52 ms).
constexpr int kMatlabThreads = 64;
template <bool DL>
__global__ void __launch_bounds__(kMatlabThreads) matlab_correct_kernel(const __grid_constant__ MatlabPairs P) {
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 32;
  const int lane = threadIdx.x % 32;
  if (w >= P.warp0[P.np]) return;
  const int k0 = matlab_problem(P, w);
  int k = k0, e = (int)(w - P.warp0[k0]);
  if (e >= min(*P.pair[k0].n_entries, P.pair[k0].max_entries)) return;
  const int* tsj = P.pair[k0].ent_tsj + 3 * (long long)e;
  const int t = tsj[0], j = tsj[2];
  const bool shared = matlab_shared(P, k0, t, j, lane);
  MatlabKey key = matlab_key(k0, tsj[1], e);
  if (shared && matlab_next(P, k0, t, j, 0, lane) != key) return;
  for (;;) {
    matlab_add_entry<DL>(P.pair[k], e, lane);
    if (!shared) return;
    key = matlab_next(P, k0, t, j, key + 1, lane);
    if (key == kNoEntry) return;
    k = (int)(key >> 60);
    e = (int)(unsigned)key;
  }
}

__global__ void min_reduce_kernel(int n, const double* __restrict__ a, double* __restrict__ out) {
  __shared__ double red[256];
  double m = 1e300;
  for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmin(m, a[i]);
  red[threadIdx.x] = m;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] = fmin(red[threadIdx.x], red[threadIdx.x + w]);
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = red[0];
}

__global__ void identity_index_kernel(int n, int* __restrict__ idx) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) idx[i] = i;
}

__global__ void add_kernel(long long n, const double* __restrict__ a, double* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] += a[i];
}


// Scratch of one candidate search: grid parameters, per-cell counts, starts
// and fill cursors, the sources sorted by cell and the largest count.
struct CandScratch {
  GridParams* gp;
  int *cell_of, *counts, *start, *fill, *sorted, *max_count;
  int cap_cells;
};

CandScratch carve_candidates(WsCarver& ws, int nt, int ns) {
  CandScratch c;
  c.cap_cells = 2 * ns + 64;
  c.gp = ws.take<GridParams>(1);
  c.cell_of = ws.take<int>((size_t)ns + 1);
  c.counts = ws.take<int>((size_t)c.cap_cells * 2 + 2);  // counts | fill cursors
  c.fill = c.counts ? c.counts + c.cap_cells + 1 : nullptr;
  c.start = ws.take<int>((size_t)c.cap_cells + 1);
  c.sorted = ws.take<int>((size_t)ns + 1);
  c.max_count = ws.take<int>(1);
  (void)nt;
  return c;
}

// Candidate lists of nt target boxes against ns source boxes (threshold thr
// on the box gap), written into nl (capacity nl->maxc per target, ascending
// source indices).  Synchronises the stream once to read the largest count:
// a non-finite curve (site 22) or a count above the capacity is reported
// here, before any list is used, with the count needed in the message and in
// ctx->last_max_cand.  *max_out receives that count.
int find_candidates(ves_ctx* c, int nt, int ns, bool same_set, const double* tbox, const double* sbox, double thr,
                    const ves_near_lists* nl, const CandScratch& cs, int* max_out, cudaStream_t s,
                    const char* what) {
  *max_out = 0;
  if (nl->maxc > 12288) {
    ves_record_error(VES_ERR_ARG, "%s: candidate capacity %d above 12288", what, nl->maxc);
    return VES_ERR_ARG;
  }
  int rc = ves_cuda_status(cudaMemsetAsync(cs.counts, 0, ((size_t)cs.cap_cells * 2 + 2) * sizeof(int), s), what);
  if (!rc) rc = ves_cuda_status(cudaMemsetAsync(cs.max_count, 0, sizeof(int), s), what);
  if (rc) return rc;
  if (ns > 0) {
    ves_count_launch(4);
    grid_setup_kernel<<<1, 1024, 0, s>>>(ns, sbox, nt, tbox, thr, cs.cap_cells, cs.gp);
    grid_count_kernel<<<ceil_div(ns, 256), 256, 0, s>>>(ns, sbox, cs.gp, cs.cell_of, cs.counts);
    scan_kernel<<<1, 1024, 0, s>>>(cs.cap_cells, cs.counts, cs.start);
    grid_fill_kernel<<<ceil_div(ns, 256), 256, 0, s>>>(ns, cs.cell_of, cs.start, cs.fill, cs.sorted);
    ves_count_launch();
    grid_candidates_kernel<<<ceil_div((long long)nt * 32, 256), 256, 0, s>>>(
        nt, same_set, tbox, sbox, thr, cs.gp, cs.start, cs.sorted, nl->maxc, nl->cand_count, nl->cand_src,
        cs.max_count);
    ves_count_launch();
    sort_candidates_kernel<<<nt, 128, (size_t)nl->maxc * sizeof(int), s>>>(nl->maxc, nl->cand_count, nl->cand_src);
  } else {
    rc = ves_cuda_status(cudaMemsetAsync(nl->cand_count, 0, (size_t)nt * sizeof(int), s), what);
    if (rc) return rc;
  }
  if ((rc = ves_launch_check(what))) return rc;
  rc = ves_cuda_status(cudaMemcpyAsync(c->h_ints, cs.max_count, sizeof(int), cudaMemcpyDeviceToHost, s), what);
  if (rc) return rc;
  if ((rc = ves_check_status(c, s, what))) {
    if (rc == VES_ERR_NONFINITE && c->h_status->where == 22)
      ves_record_error(rc, "%s: vesicle %lld has a non-finite coordinate (site 22)", what, c->h_status->aux);
    return rc;
  }
  const int mx = c->h_ints[0];
  if (mx > c->last_max_cand) c->last_max_cand = mx;
  *max_out = mx;
  if (mx > nl->maxc) {
    ves_record_error(VES_ERR_NEARLIST_OVERFLOW,
                     "%s: a vesicle has %d near-pair candidates, the lists hold %d (site 20; capacity needed %d)",
                     what, mx, nl->maxc, mx);
    return VES_ERR_NEARLIST_OVERFLOW;
  }
  return VES_OK;
}

// One MATLAB correction problem of a launch: nvt targets Xt of context ct (the
// launch's target set `set`), sources of context cs, lists nl.
MatlabPair matlab_pair(int set, const ves_ctx* ct, const ves_ctx* cs, int nvt, const double* Xt, const double* Xup_s,
                       const double* tang_up, const double* den_s, const double* vself_s, const ves_near_lists* nl,
                       double h, double* LP, double* near_only) {
  MatlabPair a;
  a.set = set;
  a.nvt = nvt;
  a.Nt = ct->N;
  a.Ns = cs->N;
  a.Nup = cs->Nup;
  a.h = h;
  a.Xt = Xt;
  a.Xup = Xup_s;
  a.tang_up = tang_up;
  a.den = den_s;
  a.vself = vself_s;
  a.lag = ct->lag;
  a.n_entries = nl->n_entries;
  a.max_entries = nl->max_entries;
  a.maxc = nl->maxc;
  a.ent_tsj = nl->ent_tsj;
  a.ent_icp = nl->ent_icp;
  a.ent_geo = nl->ent_geo;
  a.cand_count = nl->cand_count;
  a.excl_mask = nl->excl_mask;
  a.LP = LP;
  a.near_only = near_only;
  return a;
}

// The launch of np problems; index: its place, or null.  Returns the index's
// size in ints: a chain link per slot, then heads for every set of points.
size_t matlab_pairs(int np, const MatlabPair* pairs, int* index, MatlabPairs& P) {
  memset(&P, 0, sizeof(P));
  P.np = np;
  for (int k = 0; k < np; ++k) {
    P.pair[k] = pairs[k];
    P.warp0[k + 1] = P.warp0[k] + pairs[k].max_entries;
  }
  size_t n = (size_t)P.warp0[np];
  P.next = index;
  for (int k = 0; k < np; ++k) {
    int same = 0;
    while (pairs[same].set != pairs[k].set) ++same;
    if (same == k) {
      P.head[k] = index ? index + n : nullptr;
      n += (size_t)pairs[k].nvt * pairs[k].Nt;
    } else {
      P.head[k] = P.head[same];
    }
  }
  return n;
}

int make_matlab_index(int np, const MatlabPair* pairs, int* index, cudaStream_t s) {
  MatlabPairs P;
  const size_t n = matlab_pairs(np, pairs, index, P);
  const long long slots = P.warp0[np];
  if (slots <= 0) return VES_OK;
  const int rc = ves_cuda_status(cudaMemsetAsync(index + slots, 0xff, (n - slots) * sizeof(int), s), "near index");
  if (rc) return rc;
  ves_count_launch();
  matlab_index_kernel<<<ceil_div(slots, 256), 256, 0, s>>>(P);
  return ves_launch_check("near index");
}

template <bool DL>
void launch_matlab_correct(int np, const MatlabPair* pairs, const int* index, cudaStream_t s) {
  MatlabPairs P;
  matlab_pairs(np, pairs, const_cast<int*>(index), P);
  if (P.warp0[np] <= 0) return;
  ves_count_launch();
  matlab_correct_kernel<DL><<<(unsigned)ceil_div(P.warp0[np] * 32, kMatlabThreads), kMatlabThreads, 0, s>>>(P);
}

// One problem whose caller has made no index: one in `scratch` (bytes of it),
// where lists are long enough for searching them to cost more (from 4096
// entries on, 128 reads of a warp) and the scratch holds it.
template <bool DL>
int launch_matlab_correct_one(const MatlabPair& a, const int* index, void* scratch, size_t bytes, cudaStream_t s) {
  MatlabPairs P;
  if (!index && a.max_entries >= 4096 && matlab_pairs(1, &a, nullptr, P) * sizeof(int) <= bytes) {
    const int rc = make_matlab_index(1, &a, (int*)scratch, s);
    if (rc) return rc;
    index = (const int*)scratch;
  }
  launch_matlab_correct<DL>(1, &a, index, s);
  return VES_OK;
}

// The py_hh correction.  hits: hedgehog_hits of the lists, or null: made in
// scratch (3 nv N ints).
int launch_hedgehog(const ves_ctx* c, int nv, const double* X, const double* Xup, const double* vself,
                    const ves_near_lists* nl, const int* hits, int* scratch, double* LP, double* near_only,
                    cudaStream_t s) {
  if (!hits) {
    const int rc = hedgehog_hits(c, nv, nl, scratch, s);
    if (rc) return rc;
    hits = scratch;
  }
  ves_count_launch();
  hh_apply_kernel<<<nv, 128, (size_t)2 * c->N * sizeof(double), s>>>(nv, c->N, c->Nup, nl->maxc, X, Xup,
                                                                     nl->cand_count, nl->cand_src, nl->hh_mask, hits,
                                                                     vself, LP, near_only);
  return VES_OK;
}

}  // namespace

int hedgehog_hits(const ves_ctx* c, int nv, const ves_near_lists* nl, int* hits, cudaStream_t s) {
  if (nv <= 0) return VES_OK;
  const int rc = ves_cuda_status(cudaMemsetAsync(hits, 0, (size_t)nv * c->N * sizeof(int), s), "hedgehog hits");
  if (rc) return rc;
  ves_count_launch();
  hh_count_kernel<<<nv, 128, 0, s>>>(nv, c->N, c->Nup, nl->maxc, nl->cand_count, nl->cand_src, nl->hh_mask, hits);
  return ves_launch_check("hedgehog_hits");
}

int near_zone_py(ves_ctx* c, int nv, const double* X, const double* Xup_in, double thresh,
                 const ves_near_lists* nl, WsCarver& ws, cudaStream_t s) {
  const int N = c->N, Nup = c->Nup;
  double* tbox = ws.take<double>((size_t)nv * 4);
  double* sbox = ws.take<double>((size_t)nv * 4);
  double* Xup = Xup_in ? nullptr : ws.take<double>((size_t)nv * 2 * Nup);
  const CandScratch cs = carve_candidates(ws, nv, nv);
  if (ws.sizing) return VES_OK;
  if (!ws.ok()) {
    ves_record_error(VES_ERR_WORKSPACE, "near_zone_py: workspace too small");
    return VES_ERR_WORKSPACE;
  }
  if (!nl || !nl->cand_count || !nl->cand_src || !nl->excl_mask || !nl->hh_mask || nl->maxc <= 0) {
    ves_record_error(VES_ERR_ARG, "near_zone_py: incomplete near lists");
    return VES_ERR_ARG;
  }
  if (nv <= 0) return VES_OK;
  const double thr = thresh > 0 ? thresh : 1.0 / N;
  if (!Xup_in) launch_upsample(c, nv, 2, X, 2LL * N, Xup, s);
  const double* Xu = Xup_in ? Xup_in : Xup;
  ves_count_launch(2);
  bbox_kernel<<<nv, 128, 0, s>>>(N, X, tbox, c->status);
  bbox_kernel<<<nv, 128, 0, s>>>(Nup, Xu, sbox, c->status);
  int mx = 0;
  int rc = find_candidates(c, nv, nv, true, tbox, sbox, thr, nl, cs, &mx, s, "near_zone_py");
  if (rc) return rc;
  const size_t sh = (size_t)2 * N * sizeof(double) + (c->nwords_N + c->nwords_up) * sizeof(uint32_t);
  dim3 grid(mx > 0 ? mx : 1, nv);
  ves_count_launch();
  py_masks_kernel<<<grid, 256, sh, s>>>(N, Nup, nl->maxc, thr * thr, X, Xu, nl->cand_count, nl->cand_src,
                                        nl->excl_mask, nl->hh_mask);
  return ves_launch_check("near_zone_py");
}

int near_zone_matlab(ves_ctx* c, int nv, const double* X, double h, const ves_near_lists* nl, WsCarver& ws,
                     cudaStream_t s) {
  const int N = c->N;
  double* box = ws.take<double>((size_t)nv * 4);
  double* len = ws.take<double>((size_t)nv);
  double* hmin = ws.take<double>(1);
  const CandScratch cs = carve_candidates(ws, nv, nv);
  if (ws.sizing) return VES_OK;
  if (!ws.ok()) {
    ves_record_error(VES_ERR_WORKSPACE, "near_zone_matlab: workspace too small");
    return VES_ERR_WORKSPACE;
  }
  if (!nl || !nl->cand_count || !nl->cand_src || !nl->excl_mask || !nl->n_entries || !nl->ent_tsj ||
      !nl->ent_icp || !nl->ent_geo || nl->maxc <= 0) {
    ves_record_error(VES_ERR_ARG, "near_zone_matlab: incomplete near lists");
    return VES_ERR_ARG;
  }
  if (nv <= 0) return VES_OK;
  if (h <= 0) {
    launch_geom_prop(c, nv, X, nullptr, nullptr, len, s);
    ves_count_launch();
    min_reduce_kernel<<<1, 256, 0, s>>>(nv, len, hmin);
    double lmin = 0;
    int rc = ves_cuda_status(cudaMemcpyAsync(&lmin, hmin, sizeof(double), cudaMemcpyDeviceToHost, s), "hmin");
    if (!rc) rc = ves_cuda_status(cudaStreamSynchronize(s), "hmin sync");
    if (rc) return rc;
    h = lmin / N;
  }
  int rc = ves_cuda_status(cudaMemsetAsync(nl->n_entries, 0, sizeof(int), s), "zero entries");
  if (rc) return rc;
  ves_count_launch();
  bbox_kernel<<<nv, 128, 0, s>>>(N, X, box, c->status);
  int mx = 0;
  if ((rc = find_candidates(c, nv, nv, true, box, box, 2.0 * h, nl, cs, &mx, s, "near_zone_matlab"))) return rc;
  const size_t sh = (size_t)(2 * N + 49) * sizeof(double) + c->nwords_N * sizeof(uint32_t);
  dim3 grid(mx > 0 ? mx : 1, nv);
  ves_count_launch();
  matlab_zone_kernel<<<grid, 128, sh, s>>>(N, N, nl->maxc, h, X, X, c->lag, nl->cand_count, nl->cand_src,
                                           nl->excl_mask, nl->max_entries, nl->n_entries, nl->ent_tsj,
                                           nl->ent_icp, nl->ent_geo, c->status);
  return ves_launch_check("near_zone_matlab");
}

int near_sing_int_run(ves_ctx* c, int scheme, int precision, int nv, const double* X, const double* sa_up,
                      const double* Xup, const double* f, const double* vself, const ves_near_lists* nl,
                      double h, double* LP, double* near_only, WsCarver& ws, cudaStream_t s, const int* index) {
  const int N = c->N, Nup = c->Nup;
  double* fup = ws.take<double>((size_t)nv * 2 * Nup);
  double* den = ws.take<double>((size_t)nv * 2 * Nup);
  int* selfidx = ws.take<int>((size_t)nv);
  const ves_near_lists* excl = (scheme == VES_NEAR_NONE) ? nullptr : nl;
  if (ws.sizing) {
    farfield_run(c, precision, nv, Nup, Xup, den, nv, N, X, selfidx, excl, LP, ws, s);
    if (scheme == VES_NEAR_PY_RBF) rbf_near_correct(c, nv, X, f, vself, nl, LP, ws, s);
    return VES_OK;
  }
  if (!ws.ok()) {
    ves_record_error(VES_ERR_WORKSPACE, "near_sing_int: workspace too small");
    return VES_ERR_WORKSPACE;
  }
  if (scheme != VES_NEAR_NONE && scheme != VES_NEAR_PY_HH && scheme != VES_NEAR_MATLAB && scheme != VES_NEAR_PY_RBF) {
    ves_record_error(VES_ERR_ARG, "near_sing_int: bad scheme %d", scheme);
    return VES_ERR_ARG;
  }
  if (scheme != VES_NEAR_NONE && !nl) {
    ves_record_error(VES_ERR_ARG, "near_sing_int: near lists required");
    return VES_ERR_ARG;
  }
  if (nv <= 0) return VES_OK;
  if (near_only) {
    int rc0 = ves_cuda_status(cudaMemsetAsync(near_only, 0, (size_t)nv * 2 * N * sizeof(double), s), "zero near");
    if (rc0) return rc0;
  }
  if (nv == 1) {  // a single vesicle has no interactions (poten.py:485-486)
    return ves_cuda_status(cudaMemsetAsync(LP, 0, (size_t)2 * N * sizeof(double), s), "zero LP");
  }
  launch_upsample(c, nv, 2, f, 2LL * N, fup, s);
  launch_density(nv, Nup, fup, sa_up, den, s);
  ves_count_launch();
  identity_index_kernel<<<ceil_div(nv, 256), 256, 0, s>>>(nv, selfidx);
  int rc = farfield_run(c, precision, nv, Nup, Xup, den, nv, N, X, selfidx, excl, LP, ws, s);
  if (rc) return rc;
  if (scheme == VES_NEAR_PY_RBF) {
    // nearSingInt_rbf: the far field above plus the fits of the near pairs
    if ((rc = rbf_near_correct(c, nv, X, f, vself, nl, LP, ws, s))) return rc;
  } else if (scheme == VES_NEAR_PY_HH) {
    if ((rc = launch_hedgehog(c, nv, X, Xup, vself, nl, index, (int*)fup, LP, near_only, s))) return rc;
  } else if (scheme == VES_NEAR_MATLAB) {
    const MatlabPair a = matlab_pair(0, c, c, nv, X, Xup, nullptr, den, vself, nl, h, LP, near_only);
    if ((rc = launch_matlab_correct_one<false>(a, index, fup, (size_t)nv * 2 * Nup * sizeof(double), s))) return rc;
  }
  return ves_launch_check("near_sing_int");
}

// Two vesicle sets of different point counts (a mixed suspension): the near
// zone of the target points of one set w.r.t. the source vesicles of the
// other (getZone's NearOther, matlab/capsules_py.m:194-467, with the source
// set's h) and the source set's single layer at the target points with those
// entries corrected (nearSingInt with tEqualS false, matlab/poten_py.m:495-692).
int near_zone_matlab_cross(ves_ctx* ct, ves_ctx* cs, int nvt, const double* Xt, int nvs, const double* Xs, double h,
                           const ves_near_lists* nl, WsCarver& ws, cudaStream_t s) {
  const int Nt = ct->N, Ns = cs->N;
  double* tbox = ws.take<double>((size_t)nvt * 4);
  double* sbox = ws.take<double>((size_t)nvs * 4);
  const CandScratch csc = carve_candidates(ws, nvt, nvs);
  if (ws.sizing) return VES_OK;
  if (!ws.ok()) {
    ves_record_error(VES_ERR_WORKSPACE, "near_zone_cross: workspace too small");
    return VES_ERR_WORKSPACE;
  }
  if (!nl || !nl->cand_count || !nl->cand_src || !nl->excl_mask || !nl->n_entries || !nl->ent_tsj ||
      !nl->ent_icp || !nl->ent_geo || nl->maxc <= 0 || h <= 0) {
    ves_record_error(VES_ERR_ARG, "near_zone_cross: incomplete near lists or h <= 0");
    return VES_ERR_ARG;
  }
  int rc = ves_cuda_status(cudaMemsetAsync(nl->n_entries, 0, sizeof(int), s), "zero entries");
  if (rc || nvt <= 0) return rc;
  ves_count_launch(nvs > 0 ? 2 : 1);
  bbox_kernel<<<nvt, 128, 0, s>>>(Nt, Xt, tbox, ct->status);
  if (nvs > 0) bbox_kernel<<<nvs, 128, 0, s>>>(Ns, Xs, sbox, ct->status);
  int mx = 0;
  if ((rc = find_candidates(ct, nvt, nvs, false, tbox, sbox, 2.0 * h, nl, csc, &mx, s, "near_zone_cross"))) return rc;
  const size_t sh = (size_t)(2 * Ns + 49) * sizeof(double) + ct->nwords_N * sizeof(uint32_t);
  dim3 grid(mx > 0 ? mx : 1, nvt);
  ves_count_launch();
  matlab_zone_kernel<<<grid, 128, sh, s>>>(Nt, Ns, nl->maxc, h, Xt, Xs, ct->lag, nl->cand_count, nl->cand_src,
                                           nl->excl_mask, nl->max_entries, nl->n_entries, nl->ent_tsj, nl->ent_icp,
                                           nl->ent_geo, ct->status);
  return ves_launch_check("near_zone_cross");
}

// The MATLAB near-singular corrections alone (nearSingInt with the far field
// computed elsewhere, matlab/poten_py.m:495-692), several in one launch (np <=
// 16): problem k has nvt[k] targets Xt[k] of context ct[k] (target set set[k],
// LP[k] the set's), sources Xup_s[k] of context cs[k] with densities den_s[k] and self velocities vself_s[k], near
// entries nl[k], zone width h[k], and adds to LP[k].
int near_correct_matlab_pairs(int np, const int* set, ves_ctx* const* ct, ves_ctx* const* cs, const int* nvt,
                              const double* const* Xt, const double* const* Xup_s, const double* const* den_s,
                              const double* const* vself_s, const ves_near_lists* const* nl, const double* h, double* const* LP, const int* index,
                              cudaStream_t s) {
  if (np < 1 || np > kMatlabPairs) {
    ves_record_error(VES_ERR_ARG, "near_correct_matlab_pairs: 1 to %d problems", kMatlabPairs);
    return VES_ERR_ARG;
  }
  MatlabPair pairs[kMatlabPairs];
  for (int k = 0; k < np; ++k)
    pairs[k] = matlab_pair(set[k], ct[k], cs[k], nvt[k], Xt[k], Xup_s[k], nullptr, den_s[k], vself_s[k], nl[k], h[k], LP[k],
                           nullptr);
  launch_matlab_correct<false>(np, pairs, index, s);
  return ves_launch_check("near_correct_matlab_pairs");
}

size_t matlab_index_ints(int np, const int* set, ves_ctx* const* ct, const int* nvt, const ves_near_lists* const* nl) {
  MatlabPair pairs[kMatlabPairs];
  MatlabPairs P;
  for (int k = 0; k < np; ++k)
    pairs[k] = matlab_pair(set[k], ct[k], ct[k], nvt[k], nullptr, nullptr, nullptr, nullptr, nullptr, nl[k], 0.0, nullptr,
                           nullptr);
  return matlab_pairs(np, pairs, nullptr, P);
}

int matlab_index(int np, const int* set, ves_ctx* const* ct, const int* nvt, const ves_near_lists* const* nl,
                 int* index, cudaStream_t s) {
  MatlabPair pairs[kMatlabPairs];
  for (int k = 0; k < np; ++k)
    pairs[k] = matlab_pair(set[k], ct[k], ct[k], nvt[k], nullptr, nullptr, nullptr, nullptr, nullptr, nl[k], 0.0, nullptr,
                           nullptr);
  return make_matlab_index(np, pairs, index, s);
}

int near_sing_int_cross_add(ves_ctx* ct, ves_ctx* cs, int scheme, int precision, int nvt, const double* Xt, int nvs,
                            const double* Xup_s, const double* den_s, const double* vself_s,
                            const ves_near_lists* nl, double h, double* LP, WsCarver& ws, cudaStream_t s) {
  const int Nt = ct->N, Nups = cs->Nup;
  double* tmp = ws.take<double>((size_t)nvt * 2 * Nt);
  const ves_near_lists* excl = (scheme == VES_NEAR_MATLAB) ? nl : nullptr;
  if (ws.sizing) {
    farfield_run(ct, precision, nvs, Nups, Xup_s, den_s, nvt, Nt, Xt, nullptr, excl, tmp, ws, s);
    return VES_OK;
  }
  if (!ws.ok()) {
    ves_record_error(VES_ERR_WORKSPACE, "near_sing_int_cross: workspace too small");
    return VES_ERR_WORKSPACE;
  }
  if (scheme != VES_NEAR_NONE && scheme != VES_NEAR_MATLAB) {
    ves_record_error(VES_ERR_ARG, "near_sing_int_cross: scheme %d (between sets: matlab or none)", scheme);
    return VES_ERR_ARG;
  }
  if (nvt <= 0 || nvs <= 0) return VES_OK;
  int rc = farfield_run(ct, precision, nvs, Nups, Xup_s, den_s, nvt, Nt, Xt, nullptr, excl, tmp, ws, s);
  if (rc) return rc;
  const long long n = (long long)nvt * 2 * Nt;
  ves_count_launch();
  add_kernel<<<ceil_div(n, 256), 256, 0, s>>>(n, tmp, LP);
  if (scheme == VES_NEAR_MATLAB) {
    const MatlabPair a = matlab_pair(0, ct, cs, nvt, Xt, Xup_s, nullptr, den_s, vself_s, nl, h, LP, nullptr);
    if ((rc = launch_matlab_correct_one<false>(a, nullptr, tmp, (size_t)n * sizeof(double), s))) return rc;
  }
  return ves_launch_check("near_sing_int_cross");
}

// nearSingInt with kernelDirect = exactStokesDL (tstep_biem.py:236,501;
// matlab/poten_py.m:495-692): the double-layer far field over the Nup
// upsampled sources (den = fup sa_up 2pi/Nup (1 - visc)) with the near pairs
// removed, plus the correction from vself = jump f + D f: the py_hh rule
// (which uses vself only) or the MATLAB Lagrange extrapolation with the
// double layer at the Lagrange points.
int near_sing_int_dl_run(ves_ctx* c, int scheme, int precision, int nv, const double* X, const double* Xup,
                         const double* tang_up, const double* sa_up, const double* visc, const double* f,
                         const double* vself, const ves_near_lists* nl, double h, double* LP, double* near_only,
                         WsCarver& ws, cudaStream_t s, const int* index) {
  const int N = c->N, Nup = c->Nup;
  double* fup = ws.take<double>((size_t)nv * 2 * Nup);
  double* den = ws.take<double>((size_t)nv * 2 * Nup);
  int* selfidx = ws.take<int>((size_t)nv);
  const ves_near_lists* excl = (scheme == VES_NEAR_NONE) ? nullptr : nl;
  if (ws.sizing) {
    return farfield_dl_run(c, precision, nv, Nup, Xup, tang_up, den, sa_up, visc, nv, N, X, selfidx, excl, LP, ws,
                           s);
  }
  if (!ws.ok()) {
    ves_record_error(VES_ERR_WORKSPACE, "near_sing_int_dl: workspace too small");
    return VES_ERR_WORKSPACE;
  }
  if (scheme != VES_NEAR_NONE && scheme != VES_NEAR_PY_HH && scheme != VES_NEAR_MATLAB) {
    ves_record_error(VES_ERR_ARG, "near_sing_int_dl: scheme %d (the double layer supports none, py_hh, matlab)",
                     scheme);
    return VES_ERR_ARG;
  }
  if (scheme != VES_NEAR_NONE && !nl) {
    ves_record_error(VES_ERR_ARG, "near_sing_int_dl: near lists required");
    return VES_ERR_ARG;
  }
  if (nv <= 0) return VES_OK;
  if (near_only) {
    int rc0 = ves_cuda_status(cudaMemsetAsync(near_only, 0, (size_t)nv * 2 * N * sizeof(double), s), "zero near");
    if (rc0) return rc0;
  }
  if (nv == 1) return ves_cuda_status(cudaMemsetAsync(LP, 0, (size_t)2 * N * sizeof(double), s), "zero LP");
  launch_upsample(c, nv, 2, f, 2LL * N, fup, s);
  launch_dl_density(nv, Nup, fup, sa_up, visc, den, s);
  ves_count_launch();
  identity_index_kernel<<<ceil_div(nv, 256), 256, 0, s>>>(nv, selfidx);
  int rc = farfield_dl_run(c, precision, nv, Nup, Xup, tang_up, den, sa_up, visc, nv, N, X, selfidx, excl, LP, ws,
                           s);
  if (rc) return rc;
  if (scheme == VES_NEAR_PY_HH) {
    if ((rc = launch_hedgehog(c, nv, X, Xup, vself, nl, index, (int*)fup, LP, near_only, s))) return rc;
  } else if (scheme == VES_NEAR_MATLAB) {
    const MatlabPair a = matlab_pair(0, c, c, nv, X, Xup, tang_up, den, vself, nl, h, LP, near_only);
    if ((rc = launch_matlab_correct_one<true>(a, index, fup, (size_t)nv * 2 * Nup * sizeof(double), s))) return rc;
  }
  return ves_launch_check("near_sing_int_dl");
}
