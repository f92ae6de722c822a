// Batched dense algebra on per-vesicle blocks: tiled GEMM (FP64/FP32),
// GEMV, blocked LU with partial pivoting and LU solve, and the deterministic
// dot-product reduction used by GMRES.
#include "ves_internal.h"

// ----------------------------------------------------------------------------
// C[b] = alpha * A[b] (MxK) * B[b] (KxN) + beta * C[b], row-major, 64x64 tiles.
template <typename T>
__global__ void __launch_bounds__(256) bgemm_kernel(int M, int N, int K, T alpha, const T* __restrict__ A,
                                                    int lda, long long sA, const T* __restrict__ B, int ldb,
                                                    long long sB, T beta, T* __restrict__ C, int ldc,
                                                    long long sC) {
  constexpr int TM = 64, TN = 64, TK = 16;
  __shared__ T As[TK][TM + 1];
  __shared__ T Bs[TK][TN];
  const long long b = blockIdx.z;
  const T* Ab = A + b * sA;
  const T* Bb = B + b * sB;
  T* Cb = C + b * sC;
  const int row0 = blockIdx.y * TM, col0 = blockIdx.x * TN;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;  // 16x16 threads, 4x4 outputs each
  T acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = T(0);
  for (int k0 = 0; k0 < K; k0 += TK) {
    for (int idx = threadIdx.x; idx < TM * TK; idx += 256) {
      const int r = idx / TK, kk = idx % TK;
      const int gr = row0 + r, gk = k0 + kk;
      As[kk][r] = (gr < M && gk < K) ? Ab[(long long)gr * lda + gk] : T(0);
    }
    for (int idx = threadIdx.x; idx < TK * TN; idx += 256) {
      const int kk = idx / TN, cc = idx % TN;
      const int gk = k0 + kk, gc = col0 + cc;
      Bs[kk][cc] = (gk < K && gc < N) ? Bb[(long long)gk * ldb + gc] : T(0);
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < TK; ++kk) {
      T a[4], bb[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) bb[j] = Bs[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], bb[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gr = row0 + ty * 4 + i;
    if (gr >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gc = col0 + tx * 4 + j;
      if (gc >= N) continue;
      T* cp = Cb + (long long)gr * ldc + gc;
      *cp = (beta == T(0)) ? alpha * acc[i][j] : fma(alpha, acc[i][j], beta * *cp);
    }
  }
}

// FP32 variant for aligned shapes: 128x128 tiles, K steps of 8, 8x8 outputs
// per thread (rows ty*4+i and 64+ty*4+i, columns tx*4+j and 64+tx*4+j), 16-byte
// operand loads.  Needs K % 8 == 0, N % 4 == 0, lda/ldb/sA/sB multiples of 4
// and 16-byte aligned A and B.  Bound by the FP32 pipe: the next K step is
// loaded into registers while the current one is multiplied and stored into
// the other half of the shared memory, one barrier per step, and two columns'
// products are one packed FP32x2 fma (the same products in the same order).
// The Alpert products of 1024 vesicles of N = 128 (K = 1536): 45.9 -> 40.8 ms
// (49 TFLOP/s).
__global__ void __launch_bounds__(256, 2) bgemm128_f32_kernel(int M, int N, int K, float alpha,
                                                              const float* __restrict__ A, int lda, long long sA,
                                                              const float* __restrict__ B, int ldb, long long sB,
                                                              float beta, float* __restrict__ C, int ldc,
                                                              long long sC) {
  constexpr int TK = 8, LDS = 132;  // padded rows: the transposed A stores are conflict-free
  __shared__ __align__(16) float As[2][TK][LDS];
  __shared__ __align__(16) float Bs[2][TK][LDS];
  const long long b = blockIdx.z;
  const float* Ab = A + b * sA;
  const float* Bb = B + b * sB;
  float* Cb = C + b * sC;
  const int row0 = blockIdx.y * 128, col0 = blockIdx.x * 128;
  const int t = threadIdx.x, tx = t % 16, ty = t / 16;
  // load assignments: A row t/2, k chunk (t%2)*4; B row t/32, columns (t%32)*4
  const int ar = t >> 1, ak = (t & 1) * 4;
  const int bk = t >> 5, bc = (t & 31) * 4;
  const bool arow_ok = row0 + ar < M;
  const bool bcol_ok = col0 + bc < N;  // N % 4 == 0: the whole float4 is in range
  const float* ap = Ab + (long long)(arow_ok ? row0 + ar : 0) * lda + ak;
  const float* bp = Bb + (long long)bk * ldb + (bcol_ok ? col0 + bc : 0);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  auto store = [&](int buf, float4 av, float4 bv) {
    As[buf][ak + 0][ar] = av.x;
    As[buf][ak + 1][ar] = av.y;
    As[buf][ak + 2][ar] = av.z;
    As[buf][ak + 3][ar] = av.w;
    *reinterpret_cast<float4*>(&Bs[buf][bk][bc]) = bv;
  };
  float2 acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
  store(0, arow_ok ? *reinterpret_cast<const float4*>(ap) : zero, bcol_ok ? *reinterpret_cast<const float4*>(bp) : zero);
  __syncthreads();
  for (int k0 = 0, buf = 0; k0 < K; k0 += TK, buf ^= 1) {
    const bool more = k0 + TK < K;
    float4 av = zero, bv = zero;
    if (more) {
      ap += TK;
      bp += (long long)TK * ldb;
      if (arow_ok) av = *reinterpret_cast<const float4*>(ap);
      if (bcol_ok) bv = *reinterpret_cast<const float4*>(bp);
    }
#pragma unroll
    for (int kk = 0; kk < TK; ++kk) {
      const float4 a0 = *reinterpret_cast<const float4*>(&As[buf][kk][ty * 4]);
      const float4 a1 = *reinterpret_cast<const float4*>(&As[buf][kk][64 + ty * 4]);
      const float4 b0 = *reinterpret_cast<const float4*>(&Bs[buf][kk][tx * 4]);
      const float4 b1 = *reinterpret_cast<const float4*>(&Bs[buf][kk][64 + tx * 4]);
      const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const float2 bb[4] = {make_float2(b0.x, b0.y), make_float2(b0.z, b0.w), make_float2(b1.x, b1.y),
                            make_float2(b1.z, b1.w)};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = __ffma2_rn(make_float2(a[i], a[i]), bb[j], acc[i][j]);
    }
    if (more) {
      store(buf ^ 1, av, bv);
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int gr = row0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + i - 4);
    if (gr >= M) continue;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int gc = col0 + (j < 4 ? tx * 4 + j : 64 + tx * 4 + j - 4);
      if (gc >= N) continue;
      const float v = (j & 1) ? acc[i][j >> 1].y : acc[i][j >> 1].x;
      float* cp = Cb + (long long)gr * ldc + gc;
      *cp = (beta == 0.f) ? alpha * v : fmaf(alpha, v, beta * *cp);
    }
  }
}

template <typename T>
static void bgemm_launch(int batch, int M, int N, int K, T alpha, const T* A, int lda, long long sA,
                         const T* B, int ldb, long long sB, T beta, T* C, int ldc, long long sC,
                         cudaStream_t s) {
  for (int b0 = 0; b0 < batch; b0 += 65535) {
    const int nb = batch - b0 < 65535 ? batch - b0 : 65535;
    dim3 grid(ceil_div(N, 64), ceil_div(M, 64), nb);
    ves_count_launch();
    bgemm_kernel<T><<<grid, 256, 0, s>>>(M, N, K, alpha, A + b0 * sA, lda, sA, B + b0 * sB, ldb, sB, beta,
                                         C + b0 * sC, ldc, sC);
  }
}

void launch_bgemm_f64(int batch, int M, int N, int K, double alpha, const double* A, int lda,
                      long long sA, const double* B, int ldb, long long sB, double beta, double* C,
                      int ldc, long long sC, cudaStream_t s) {
  bgemm_launch<double>(batch, M, N, K, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, s);
}
void launch_bgemm_f32(int batch, int M, int N, int K, float alpha, const float* A, int lda,
                      long long sA, const float* B, int ldb, long long sB, float beta, float* C,
                      int ldc, long long sC, cudaStream_t s) {
  const bool aligned = K % 8 == 0 && N % 4 == 0 && lda % 4 == 0 && ldb % 4 == 0 && sA % 4 == 0 && sB % 4 == 0 &&
                       ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15u) == 0;
  if (!aligned || M < 64) {
    bgemm_launch<float>(batch, M, N, K, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, s);
    return;
  }
  for (int b0 = 0; b0 < batch; b0 += 65535) {
    const int nb = batch - b0 < 65535 ? batch - b0 : 65535;
    dim3 grid(ceil_div(N, 128), ceil_div(M, 128), nb);
    ves_count_launch();
    bgemm128_f32_kernel<<<grid, 256, 0, s>>>(M, N, K, alpha, A + b0 * sA, lda, sA, B + b0 * sB, ldb, sB, beta,
                                             C + b0 * sC, ldc, sC);
  }
}

// ----------------------------------------------------------------------------
// Sums over the warp of four values per lane, in the order of the usual
// exchange (lanes 16 apart, then 8, 4, 2, 1): the lanes 8 q .. 8 q + 7 get the
// sum of s[q].  The first two exchanges add different values in the two halves
// and quarters of the warp, so the four sums take 6 additions.
__device__ __forceinline__ double warp_sum4(const double* s, int lane) {
  const bool h = lane & 16, f = lane & 8;
  const double u0 = (h ? s[2] : s[0]) + __shfl_xor_sync(0xffffffffu, h ? s[0] : s[2], 16);
  const double u1 = (h ? s[3] : s[1]) + __shfl_xor_sync(0xffffffffu, h ? s[1] : s[3], 16);
  double t = (f ? u1 : u0) + __shfl_xor_sync(0xffffffffu, f ? u0 : u1, 8);
  t += __shfl_xor_sync(0xffffffffu, t, 4);
  t += __shfl_xor_sync(0xffffffffu, t, 2);
  t += __shfl_xor_sync(0xffffffffu, t, 1);
  return t;
}

// y[k] = A[k] (m x n) x[k]; one CTA per vesicle, four rows to a warp (bound by
// the FP64 pipe: one row's own reduction cost 5 additions next to n/32
// multiply-adds; 1024 blocks of 256 rows 0.205 -> 0.147 ms).
__global__ void __launch_bounds__(256) bgemv_kernel(int m, int n, const double* __restrict__ A,
                                                    const double* __restrict__ x, long long xs,
                                                    double* __restrict__ y, long long ys) {
  extern __shared__ double xsh[];
  const int k = blockIdx.x;
  for (int i = threadIdx.x; i < n; i += blockDim.x) xsh[i] = x[(long long)k * xs + i];
  __syncthreads();
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, nw = blockDim.x / 32;
  const double* Ak = A + (long long)k * m * n;
  for (int r = 4 * warp; r < m; r += 4 * nw) {
    const double* row = Ak + (long long)r * n;
    const int mr = min(4, m - r);
    const long long s1 = mr > 1 ? n : 0, s2 = mr > 2 ? 2LL * n : 0, s3 = mr > 3 ? 3LL * n : 0;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
    for (int c = lane; c < n; c += 32) {
      const double v = xsh[c];
      s[0] = fma(row[c], v, s[0]);
      s[1] = fma(row[s1 + c], v, s[1]);
      s[2] = fma(row[s2 + c], v, s[2]);
      s[3] = fma(row[s3 + c], v, s[3]);
    }
    const double t = warp_sum4(s, lane);
    const int q = lane >> 3;
    if ((lane & 7) == 0 && q < mr) y[(long long)k * ys + r + q] = t;
  }
}

void launch_bgemv_f64(int nv, int m, int n, const double* A, const double* x, long long xs, double* y,
                      long long ys, cudaStream_t s) {
  if (nv <= 0) return;
  ves_count_launch();
  bgemv_kernel<<<nv, 256, (size_t)n * sizeof(double), s>>>(m, n, A, x, xs, y, ys);
}

// ----------------------------------------------------------------------------
// Blocked right-looking LU with partial pivoting, one CTA per matrix
// (the factorisation torch.linalg.lu_factor performs, tstep_biem.py:350).
// piv[j] = row exchanged with row j at step j (LAPACK ipiv, 0-based).
//
// Panels of 32 columns.  A thread keeps ROWS whole rows of the panel in
// registers, so a column costs two barriers: one for the largest entry (the
// first on ties), one for the pivot row and the row it replaces, which pass
// through shared memory.  Eight columns are unrolled (32 make 200 KB of
// instructions, and fetching them was the bound), then they move to shared
// memory, where the panel lies transposed (Lt) for what follows.  The panel's
// row exchanges are worked out as one permutation: every other column is read, permuted and, right of the panel,
// solved against the unit triangle by one thread, and the trailing matrix is
// updated in 32 x 32 tiles per warp, 8 x 4 entries per thread.  An entry takes
// its multiply-adds in ascending order of the column eliminated, whatever the
// tiles, so the factors do not depend on them.
// FP64 is bound by its pipe (1000 matrices of 384: 19 G multiply-adds, 33 ms;
// 46.9 -> 39.3 ms; 8192 of 96: 4.1 ms, 9.1 -> 7.0), FP32 by the latency of a
// column (1024 of 384: 13.8 -> 3.5 ms).
constexpr int LU_NB = 32;

// distance of the transposed panel's rows: 16-byte aligned, off a multiple of 16
__host__ __device__ inline int lu_pitch(int n) {
  const int np = (n + 3) / 4 * 4;
  return np % 16 ? np : np + 4;
}

template <typename T>
__device__ __forceinline__ void lu_ld4(const T* p, T* v) {
  if constexpr (sizeof(T) == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
  } else {
    const double2 t = reinterpret_cast<const double2*>(p)[0], u = reinterpret_cast<const double2*>(p)[1];
    v[0] = t.x, v[1] = t.y, v[2] = u.x, v[3] = u.y;
  }
}
template <typename T>
__device__ __forceinline__ void lu_st4(T* p, const T* v) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
    reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
    reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
  }
}

// |x| as an integer of the same order, -1 for a NaN: comparing FP64 values
// would take the FP64 pipe
__device__ __forceinline__ int lu_key(float x) {
  const int b = __float_as_int(x) & 0x7fffffff;
  return b > 0x7f800000 ? -1 : b;
}
__device__ __forceinline__ long long lu_key(double x) {
  const long long b = __double_as_longlong(x) & 0x7fffffffffffffffLL;
  return b > 0x7ff0000000000000LL ? -1 : b;
}

template <typename T, int ROWS, int NT, int CTAS>
__global__ void __launch_bounds__(NT, CTAS) lu_factor_kernel(int n, T* __restrict__ A, int* __restrict__ piv,
                                                             VesDeviceStatus* st) {
  constexpr int NB = LU_NB, NW = NT / 32;
  using Key = decltype(lu_key(T(0)));
  extern __shared__ __align__(16) unsigned char lu_sh[];
  const int np = lu_pitch(n);
  T* Lt = (T*)lu_sh;        // [NB][np] the panel, transposed
  T* U12 = Lt + NB * np;    // [NB][np] the panel's rows of the other columns
  __shared__ __align__(16) T prow[NB], jrow[NB];
  __shared__ Key wv[NW];
  __shared__ T pinv;
  __shared__ int wi[NW], lpiv[NB], top[NB], orow[NB], osrc[NB], ocnt;
  const int k = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  T* a = A + (long long)k * n * n;
  int* pv = piv + (long long)k * n;
  const bool vec = n % 4 == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;

  for (int p0 = 0; p0 < n; p0 += NB) {
    const int nb = min(NB, n - p0), rows = n - p0;
    for (int i = warp; i < rows; i += NW)
      if (lane < nb) Lt[lane * np + i] = a[(long long)(p0 + i) * n + p0 + lane];
    __syncthreads();
    T row[ROWS][NB];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const int i = tid + r * NT;
#pragma unroll
      for (int j = 0; j < NB; ++j) row[r][j] = (i < rows && j < nb) ? Lt[j * np + i] : T(0);
    }
    // eight columns per pass: the registers hold columns j0 .. j0 + 31 (those
    // past the panel are zero)
#pragma unroll 1
    for (int j0 = 0; j0 < nb; j0 += 8) {
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) {
        const int j = j0 + jj;
        if (j >= nb) break;
        // pivot: first index of max |a_ij|, i >= j (a NaN is never the largest)
        Key best = -1;
        int bi = j;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          const int i = tid + r * NT;
          const Key v = lu_key(row[r][jj]);
          if (i >= j && i < rows && v > best) {
            best = v;
            bi = i;
          }
        }
        for (int o = 16; o > 0; o >>= 1) {
          const Key v2 = __shfl_xor_sync(0xffffffffu, best, o);
          const int i2 = __shfl_xor_sync(0xffffffffu, bi, o);
          if (v2 > best || (v2 == best && i2 < bi)) {
            best = v2;
            bi = i2;
          }
        }
        if (lane == 0) {
          wv[warp] = best;
          wi[warp] = bi;
        }
        __syncthreads();
        best = wv[0];
        int ip = wi[0];
#pragma unroll
        for (int w = 1; w < NW; ++w) {
          const Key v2 = wv[w];
          const int i2 = wi[w];
          if (v2 > best || (v2 == best && i2 < ip)) {
            best = v2;
            ip = i2;
          }
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          const int i = tid + r * NT;
          if (i == ip) {
#pragma unroll
            for (int q = 0; q < NB; q += 4) lu_st4(prow + q, &row[r][q]);
            pinv = (row[r][jj] != T(0)) ? T(1) / row[r][jj] : T(0);
          }
          if (i == j && ip != j) {
#pragma unroll
            for (int q = 0; q < NB; q += 4) lu_st4(jrow + q, &row[r][q]);
          }
        }
        if (tid == 0) {
          lpiv[j] = ip;
          pv[p0 + j] = p0 + ip;
          if (best == 0) ves_set_error(st, VES_ERR_SINGULAR, 1, (long long)k * n + p0 + j);
        }
        __syncthreads();
        if (ip != j && tid < j0) {  // the columns already in shared memory
          const T t = Lt[tid * np + ip];
          Lt[tid * np + ip] = Lt[tid * np + j];
          Lt[tid * np + j] = t;
        }
        const T rcp = pinv;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          const int i = tid + r * NT;
          if (ip != j && (i == ip || i == j)) {
            const T* from = i == ip ? jrow : prow;
#pragma unroll
            for (int q = 0; q < NB; q += 4) lu_ld4(from + q, &row[r][q]);
          }
          if (i > j && i < rows) {
            const T l = row[r][jj] * rcp;
            row[r][jj] = l;
#pragma unroll
            for (int g = 0; g < NB; g += 8) {
              if (g > 0 && j0 + g >= nb) break;
#pragma unroll
              for (int q = g; q < g + 8; q += 4) {
                T u[4];
                lu_ld4(prow + q, u);
#pragma unroll
                for (int e = 0; e < 4; ++e)
                  if (q + e > jj) row[r][q + e] = fma(-l, u[e], row[r][q + e]);
              }
            }
          }
        }
      }
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const int i = tid + r * NT;
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (i < rows && j0 + q < nb) Lt[(j0 + q) * np + i] = row[r][q];
#pragma unroll
        for (int q = 0; q < NB; ++q) row[r][q] = q + 8 < NB ? row[r][q + 8] : T(0);
      }
    }
    __syncthreads();
    // the nb exchanges as one permutation: top[j] = row that ends at place j,
    // orow / osrc = rows below the panel's that change and what they receive
    // (always one of the panel's own rows: place j takes a lower row only at
    // step j, after which no exchange moves it down)
    if (warp == 0) {
      int t = lane, orw = -1, osr = -1, cnt = 0;
      for (int j = 0; j < nb; ++j) {
        const int r2 = lpiv[j];
        const int tj = __shfl_sync(0xffffffffu, t, j);
        if (r2 < nb) {
          const int t2 = __shfl_sync(0xffffffffu, t, r2);
          if (lane == r2) t = tj;
          if (lane == j) t = t2;
        } else {
          const unsigned m = __ballot_sync(0xffffffffu, orw == r2);
          const int e = m ? __ffs(m) - 1 : cnt;
          if (!m && lane == cnt) orw = osr = r2;
          if (!m) ++cnt;
          const int oe = __shfl_sync(0xffffffffu, osr, e);
          if (lane == j) t = oe;
          if (lane == e) osr = tj;
        }
      }
      top[lane] = t;
      orow[lane] = orw;
      osrc[lane] = osr;
      if (lane == 0) ocnt = cnt;
    }
    __syncthreads();
    for (int i = warp; i < rows; i += NW)
      if (lane < nb) a[(long long)(p0 + i) * n + p0 + lane] = Lt[lane * np + i];
    // the other columns, one thread each
    for (int c = tid; c < n; c += NT) {
      if (c >= p0 && c < p0 + nb) continue;
      T col[NB];
      T* ac = a + (long long)p0 * n + c;
#pragma unroll
      for (int j = 0; j < NB; ++j) col[j] = j < nb ? ac[(long long)j * n] : T(0);
#pragma unroll
      for (int j = 0; j < NB; ++j)
        if (j < nb) U12[j * np + c] = col[j];
#pragma unroll
      for (int j = 0; j < NB; ++j)
        if (j < nb) col[j] = top[j] < nb ? U12[top[j] * np + c] : ac[(long long)top[j] * n];
      for (int e = 0; e < ocnt; ++e) ac[(long long)orow[e] * n] = U12[osrc[e] * np + c];
      if (c > p0) {  // L11^{-1} A12; nb == NB
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          const T v = col[j];
#pragma unroll
          for (int q = j / 4 * 4; q < NB; q += 4) {
            T l[4];
            lu_ld4(Lt + j * np + q, l);
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (q + e > j) col[q + e] = fma(-l[e], v, col[q + e]);
          }
          U12[j * np + c] = v;
        }
      }
#pragma unroll
      for (int j = 0; j < NB; ++j)
        if (j < nb) ac[(long long)j * n] = col[j];
    }
    __syncthreads();
    // A22 -= L21 U12; the tiles' last rows and columns may lie past the matrix:
    // their operands are whatever follows in shared memory, and are not stored
    const int m2 = rows - nb, nr = (m2 + 31) / 32;
    const int ty = lane >> 3, tx = lane & 7;
    for (int u = warp; u < nr * nr; u += NW) {
      const int i0 = u / nr * 32 + 8 * ty, c0 = u % nr * 32 + 4 * tx;  // in A22
      T* at = a + (long long)(p0 + nb + i0) * n + p0 + nb + c0;
      const int mr = min(8, m2 - i0), mc = min(4, m2 - c0);
      T acc[8][4];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        if (r < mr && vec && mc > 0) {
          lu_ld4(at + (long long)r * n, acc[r]);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[r][e] = (r < mr && e < mc) ? at[(long long)r * n + e] : T(0);
        }
      }
      const T* lp = Lt + nb + i0;
      const T* up = U12 + p0 + nb + c0;
#pragma unroll 4
      for (int j = 0; j < NB; ++j) {
        T l[8], v[4];
        lu_ld4(lp + j * np, l);
        lu_ld4(lp + j * np + 4, l + 4);
        lu_ld4(up + j * np, v);
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[r][e] = fma(-l[r], v[e], acc[r][e]);
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        if (r < mr && vec && mc > 0) {
          lu_st4(at + (long long)r * n, acc[r]);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (r < mr && e < mc) at[(long long)r * n + e] = acc[r][e];
        }
      }
    }
    __syncthreads();
  }
}

template <typename T, int ROWS, int NT, int CTAS>
static int lu_factor_start(ves_ctx* c, int nv, int n, T* A, int* piv, cudaStream_t s) {
  const size_t sh = ((size_t)2 * LU_NB * lu_pitch(n) + 32) * sizeof(T);  // the last tiles read up to 31 past the end
  if (sh > 32 * 1024) {  // dynamic + static shared memory must fit the opt-in limit
    int rc = ves_cuda_status(
        cudaFuncSetAttribute(lu_factor_kernel<T, ROWS, NT, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh),
        "lu_factor smem attribute");
    if (rc) return rc;
  }
  ves_count_launch();
  lu_factor_kernel<T, ROWS, NT, CTAS><<<nv, NT, sh, s>>>(n, A, piv, c->status);
  return ves_launch_check("lu_factor");
}

template <typename T>
static int lu_factor_t(ves_ctx* c, int nv, int n, T* A, int* piv, cudaStream_t s) {
  if (nv <= 0) return VES_OK;
  if ((size_t)2 * LU_NB * n * sizeof(T) > 220 * 1024) {
    ves_record_error(VES_ERR_SHAPE, "lu_factor: n=%d too large", n);
    return VES_ERR_SHAPE;
  }
  // a thread per panel row, or two or four rows per thread where a CTA has
  // fewer threads; FP64 stops at n = 440
  if (n <= 128) return lu_factor_start<T, 1, 128, 4>(c, nv, n, A, piv, s);
  if (n <= 256) return lu_factor_start<T, 1, 256, 2>(c, nv, n, A, piv, s);
  if constexpr (sizeof(T) == 8) {
    return lu_factor_start<T, 2, 256, 1>(c, nv, n, A, piv, s);
  } else {
    if (n <= 512) return lu_factor_start<T, 2, 256, 2>(c, nv, n, A, piv, s);
    return lu_factor_start<T, 4, 256, 1>(c, nv, n, A, piv, s);
  }
}

int launch_lu_factor(ves_ctx* c, int nv, int n, double* A, int* piv, cudaStream_t s) {
  return lu_factor_t<double>(c, nv, n, A, piv, s);
}

int launch_lu_factor_f32(ves_ctx* c, int nv, int n, float* A, int* piv, cudaStream_t s) {
  return lu_factor_t<float>(c, nv, n, A, piv, s);
}

// x = LU^{-1} P b per vesicle, one CTA each.  Blocks of 32 rows: the
// off-diagonal part is a GEMV, four rows to a warp, the 32x32 diagonal block
// is solved by one warp.  Bound by the FP64 pipe (16 cycles per warp
// instruction): n^2 multiply-adds, plus what each row's reduction, each
// conversion of an FP32 factor and each division cost there.  So four rows are
// reduced together (6 additions instead of 20), factors are widened by integer
// operations, and a division by a diagonal entry is a product with its
// reciprocal, taken for the whole block at once, and Markstein's correction
// (two multiply-adds, correctly rounded when the reciprocal is; IBM J. Res.
// Dev. 34, 1990).  The row exchanges walk the pivots in shared memory.  One
// solve: 1024 blocks of 384 rows in FP32 1.22 -> 0.71 ms, 301 of 192 in FP64
// 0.21 -> 0.11, 16 of 96 0.075 -> 0.040.
template <typename T>
__global__ void __launch_bounds__(256) lu_solve_kernel(int n, const T* __restrict__ LU,
                                                       const int* __restrict__ piv,
                                                       const double* __restrict__ b, double* __restrict__ x) {
  extern __shared__ double xs[];  // [n], then the pivots [n]
  __shared__ double tile[32][33], rcp[32];
  int* pv = reinterpret_cast<int*>(xs + n);
  const int k = blockIdx.x;
  const T* a = LU + (long long)k * n * n;
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  for (int i = tid; i < n; i += blockDim.x) {
    xs[i] = b[(long long)k * n + i];
    pv[i] = piv[(long long)k * n + i];
  }
  __syncthreads();
  if (tid == 0) {
    for (int j = 0; j < n; ++j) {
      const int p = pv[j];
      if (p != j) {
        const double t = xs[j];
        xs[j] = xs[p];
        xs[p] = t;
      }
    }
  }
  __syncthreads();
  // xs[r] -= sum_{c0 <= c < c1} a[r][c] xs[c] for the rows r0 .. r0 + nr - 1
  // (lane l sums the columns c0 + l, + 32, ..., then the lanes meet pairwise)
  auto off_diagonal = [&](int r0, int nr, int c0, int c1) {
    const int rr = 4 * warp;
    if (c0 >= c1 || rr >= nr) return;
    const T* row = a + (long long)(r0 + rr) * n;
    const int m = min(4, nr - rr);
    const long long s1 = m > 1 ? n : 0, s2 = m > 2 ? 2LL * n : 0, s3 = m > 3 ? 3LL * n : 0;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
    for (int c = c0 + lane; c < c1; c += 32) {
      const T a0 = row[c], a1 = row[s1 + c], a2 = row[s2 + c], a3 = row[s3 + c];
      const double v = xs[c];
      s[0] = fma(widen(a0), v, s[0]);
      s[1] = fma(widen(a1), v, s[1]);
      s[2] = fma(widen(a2), v, s[2]);
      s[3] = fma(widen(a3), v, s[3]);
    }
    const double t = warp_sum4(s, lane);
    const int q = lane >> 3;
    if ((lane & 7) == 0 && q < m) xs[r0 + rr + q] -= t;
  };
  auto load_tile = [&](int r0, int nr) {
    for (int i = tid; i < nr * 32; i += blockDim.x) {
      const int r = i >> 5, c = i & 31;
      if (c < nr) tile[r][c] = widen(a[(long long)(r0 + r) * n + r0 + c]);
    }
  };
  // forward: unit lower
  for (int r0 = 0; r0 < n; r0 += 32) {
    const int nr = min(32, n - r0);
    load_tile(r0, nr);
    off_diagonal(r0, nr, 0, r0);
    __syncthreads();
    if (warp == 0) {
      double v = (lane < nr) ? xs[r0 + lane] : 0.0;
      for (int j = 0; j < nr; ++j) {
        const double xj = __shfl_sync(0xffffffffu, v, j);
        if (lane > j && lane < nr) v = fma(-tile[lane][j], xj, v);
      }
      if (lane < nr) xs[r0 + lane] = v;
    }
    __syncthreads();
  }
  // backward: upper
  for (int r1 = n; r1 > 0; r1 -= 32) {
    const int r0 = max(0, r1 - 32), nr = r1 - r0;
    load_tile(r0, nr);
    off_diagonal(r0, nr, r1, n);
    if (warp == 7) rcp[lane] = lane < nr ? 1.0 / widen(a[(long long)(r0 + lane) * n + r0 + lane]) : 1.0;
    __syncthreads();
    if (warp == 0) {
      double v = (lane < nr) ? xs[r0 + lane] : 0.0;
      for (int j = nr - 1; j >= 0; --j) {
        const double vj = __shfl_sync(0xffffffffu, v, j), d = tile[j][j], y = rcp[j];
        const double xj = quotient(vj, d, y);
        if (lane == j) v = xj;
        if (lane < j) v = fma(-tile[lane][j], xj, v);
      }
      if (lane < nr) xs[r0 + lane] = v;
    }
    __syncthreads();
  }
  for (int i = tid; i < n; i += blockDim.x) x[(long long)k * n + i] = xs[i];
}

void launch_lu_solve(int nv, int n, const double* LU, const int* piv, const double* b, double* x,
                     cudaStream_t s) {
  if (nv <= 0) return;
  ves_count_launch();
  lu_solve_kernel<double><<<nv, 256, (size_t)n * (sizeof(double) + sizeof(int)), s>>>(n, LU, piv, b, x);
}

// the same solve with an FP32 factorisation (FP64 right-hand side, FP64 sums)
void launch_lu_solve_f32(int nv, int n, const float* LU, const int* piv, const double* b, double* x,
                         cudaStream_t s) {
  if (nv <= 0) return;
  ves_count_launch();
  lu_solve_kernel<float><<<nv, 256, (size_t)n * (sizeof(double) + sizeof(int)), s>>>(n, LU, piv, b, x);
}

// ----------------------------------------------------------------------------
// Deterministic dot product: fixed number of blocks, fixed reduction order.
constexpr int DOT_BLOCKS = 512;
int dot_partial_blocks() { return DOT_BLOCKS; }

__global__ void __launch_bounds__(256) dot_partials_kernel(long long n, const double* __restrict__ a,
                                                           const double* __restrict__ b,
                                                           double* __restrict__ partials) {
  __shared__ double red[256];
  double s = 0.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    s = fma(a[i], b[i], s);
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) partials[blockIdx.x] = red[0];
}

void launch_dot_partials(long long n, const double* a, const double* b, double* partials, cudaStream_t s) {
  ves_count_launch();
  dot_partials_kernel<<<DOT_BLOCKS, 256, 0, s>>>(n, a, b, partials);
}
