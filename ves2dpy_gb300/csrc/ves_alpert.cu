// Alpert log-singular single-layer matrix (Poten.stokesSLmatrix,
// mytorch/poten.py:40-99, weights poten.py:899-974).
//
// For target s of the Nup-upsampled curve the quadrature has 14 off-grid
// nodes (7 on each side, at offsets +-v_q*h) whose positions come from the
// trig interpolant, and Nup-9 on-grid nodes s+i, i = 5..Nup-5.  With
// F_q(s) = w_q * {1/2 log rho, dx^2 rho, dx dy rho, dy^2 rho},
// rho = 1/(|x_s - node|^2 + 1e-7), the row of the Nup x Nup matrix is
//   W(s, i) = [5 <= i <= Nup-5] F_{i+2}(s) + sum_{dense q} A_q(i) F_q(s),
//   Gup[s][(s+i) mod Nup] = sa_up[(s+i) mod Nup] * W(s, i),
// and G = R * Gup * P restricts it to the N-point grid.
#include <algorithm>

#include "ves_fft.cuh"
#include "ves_internal.h"

template <typename T>
__device__ __forceinline__ T tlog(T x);
template <>
__device__ __forceinline__ float tlog<float>(float x) { return logf(x); }
template <>
__device__ __forceinline__ double tlog<double>(double x) { return log(x); }

// FP64 -> T, and 1 / x for the kernel's regularised square distances
template <typename T>
__device__ __forceinline__ T to(double x);
template <>
__device__ __forceinline__ float to<float>(double x) { return narrow(x); }
template <>
__device__ __forceinline__ double to<double>(double x) { return x; }
__device__ __forceinline__ float inverse(float x) { return x >= kRcpMin && x <= kRcpMax ? rcp_normal(x) : 1.0f / x; }
__device__ __forceinline__ double inverse(double x) { return 1.0 / x; }

// Kernel A: per (vesicle, target s) the 14 off-grid node field values.
template <typename T>
__global__ void alpert_dense_nodes_kernel(int N, int Nup, int m, int nquad, const double* __restrict__ X,
                                          const double* __restrict__ Xup, const double* __restrict__ cq,
                                          const double* __restrict__ qw, T* __restrict__ Fd) {
  extern __shared__ double sh[];
  double* x = sh;
  double* y = x + N;
  const int k = blockIdx.y;
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    x[i] = X[(long long)k * 2 * N + i];
    y[i] = X[(long long)k * 2 * N + N + i];
  }
  __syncthreads();
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= Nup) return;
  const double xs = Xup[(long long)k * 2 * Nup + s], ys = Xup[(long long)k * 2 * Nup + Nup + s];
  T* out = Fd + ((long long)k * Nup + s) * 56;
  for (int q = 0; q < 14; ++q) {
    const double* cr = cq + (long long)q * Nup;
    double nx = 0, ny = 0;
    int r = s;
    for (int i = 0; i < N; ++i) {
      nx = fma(cr[r], x[i], nx);
      ny = fma(cr[r], y[i], ny);
      r -= m;
      if (r < 0) r += Nup;
    }
    const T dx = (T)(xs - nx), dy = (T)(ys - ny);
    const T rho = T(1) / (dx * dx + dy * dy + T(1e-7));
    const T w = (T)(q < 7 ? qw[q] : qw[nquad - 14 + q]);
    out[q * 4 + 0] = T(0.5) * w * tlog<T>(rho);
    out[q * 4 + 1] = w * dx * dx * rho;
    out[q * 4 + 2] = w * dx * dy * rho;
    out[q * 4 + 3] = w * dy * dy * rho;
  }
}

// Kernel B: rows of Gup (three fields G11, G12, G22) for ROWS targets per CTA.
// In FP32 an entry is 28 packed multiply-adds, a logarithm, a reciprocal and two
// FP64 differences; those, 32 cycles of the FP64 pipe per warp, bound it from
// below (0.57 ms for 73 vesicles of Nup = 1536), instruction issue does now.
// The conversions to FP32 took 48 cycles more there, so they are done in
// integers, the jacobian's once per CTA, and the division is branch-free: 1.55
// -> 1.14 ms.  One column per thread and one row at a time, 36 warps per SM: two
// or three columns or eight rows in flight need registers that cost more warps
// than they save loads (1.25 .. 1.8 ms).
template <typename T, int ROWS, int THREADS, int CTAS>
__global__ void __launch_bounds__(THREADS, CTAS) alpert_rows_kernel(int Nup, int nquad,
                                                                    const double* __restrict__ Xup,
                                                                    const double* __restrict__ sa_up,
                                                                    const T* __restrict__ adense,
                                                                    const double* __restrict__ qw,
                                                                    const T* __restrict__ Fd, T* __restrict__ Gup,
                                                                    int k0) {
  __shared__ __align__(16) T fd[ROWS][56];
  __shared__ double txs[ROWS], tys[ROWS];
  extern __shared__ float saf[];    // [Nup], FP32 only
  const int kl = blockIdx.y;        // vesicle within chunk
  const int k = k0 + kl;            // global vesicle
  const int s0 = blockIdx.x * ROWS;
  const double* xk = Xup + (long long)k * 2 * Nup;
  const double* sak = sa_up + (long long)k * Nup;
  for (int idx = threadIdx.x; idx < ROWS * 56; idx += THREADS) {
    const int r = idx / 56, e = idx % 56;
    fd[r][e] = (s0 + r < Nup) ? Fd[((long long)k * Nup + s0 + r) * 56 + e] : T(0);
  }
  if (threadIdx.x < ROWS) {
    const int s = min(s0 + (int)threadIdx.x, Nup - 1);
    txs[threadIdx.x] = xk[s];
    tys[threadIdx.x] = xk[Nup + s];
  }
  if (sizeof(T) == 4)
    for (int i = threadIdx.x; i < Nup; i += THREADS) saf[i] = narrow(sak[i]);
  __syncthreads();
  const T wg = (T)qw[7];  // on-grid weight h/(4 pi)
  const long long NN = (long long)Nup * Nup;
  T* G11 = Gup + (long long)kl * 3 * NN;
  T* G12 = G11 + NN;
  T* G22 = G12 + NN;
  for (int i = threadIdx.x; i < Nup; i += THREADS) {
    T a[14];
#pragma unroll
    for (int q = 0; q < 14; ++q) a[q] = adense[(long long)q * Nup + i];
    const bool grid = (i >= 5 && i <= Nup - 5);
#pragma unroll(sizeof(T) == 4 ? 1 : ROWS)
    for (int r = 0; r < ROWS; ++r) {
      const int s = s0 + r;
      if (s >= Nup) break;
      T wl = 0, wxx = 0, wxy = 0, wyy = 0;
      if constexpr (sizeof(T) == 4) {
        float2 w0 = make_float2(0.f, 0.f), w1 = w0;
#pragma unroll
        for (int q = 0; q < 14; ++q) {
          const float4 f = *reinterpret_cast<const float4*>(&fd[r][q * 4]);
          const float2 aa = make_float2(a[q], a[q]);
          w0 = __ffma2_rn(aa, make_float2(f.x, f.y), w0);
          w1 = __ffma2_rn(aa, make_float2(f.z, f.w), w1);
        }
        wl = w0.x;
        wxx = w0.y;
        wxy = w1.x;
        wyy = w1.y;
      } else {
#pragma unroll
        for (int q = 0; q < 14; ++q) {
          wl += a[q] * fd[r][q * 4 + 0];
          wxx += a[q] * fd[r][q * 4 + 1];
          wxy += a[q] * fd[r][q * 4 + 2];
          wyy += a[q] * fd[r][q * 4 + 3];
        }
      }
      int col = s + i;
      if (col >= Nup) col -= Nup;
      if (grid) {
        const T dx = to<T>(txs[r] - xk[col]), dy = to<T>(tys[r] - xk[Nup + col]);
        const T rho = inverse(dx * dx + dy * dy + T(1e-7));
        wl += T(0.5) * wg * tlog<T>(rho);
        wxx += wg * dx * dx * rho;
        wxy += wg * dx * dy * rho;
        wyy += wg * dy * dy * rho;
      }
      const T sa = sizeof(T) == 4 ? (T)saf[col] : (T)sak[col];
      const long long o = (long long)s * Nup + col;
      G11[o] = (wl + wxx) * sa;
      G12[o] = wxy * sa;
      G22[o] = (wl + wyy) * sa;
    }
  }
}

// The products with the interpolation matrices P (Nup x N) and R = (N / Nup)
// P^T in FP64, as transforms.  A row g of length Nup = m N times P is its
// Fourier coefficients of frequency |k| <= N/2 (the two at +-N/2 averaged)
// evaluated on the N grid:
//   (g P)[i] = 1/N sum_k c_k e^(-2 pi i k i / N) sum_r e^(2 pi i k r / Nup) Z_r[k],
//   Z_r[k] = sum_q g[m q + r] e^(2 pi i k q / N),
// so m transforms of length N, m N multiply-adds and one transform back: ~16k
// FP64 instructions per row at N = 96 where the dense product's row takes 92k,
// and FP64 is what bounds it (200 vesicles: 131 -> 18 ms for both products).  Two real rows make one complex sequence; a CTA
// takes ``pairs`` of them.  The result is written transposed, out[b][i][row],
// so that the same kernel applied to it gives the product with P^T.
//
// One radix-2 pass over ``nseq`` sequences of length N = R P (R = 1 or 3, P a
// power of two) whose subsequences sit in bit-reversed order; table step
// ``ts`` = Nup / N.
__device__ __forceinline__ void seq_fft(double2* z, int nseq, int N, const double* __restrict__ cs,
                                        const double* __restrict__ sn, double sign, int ts) {
  const int R = (N % 3 == 0) ? 3 : 1, P = N / R, half = P / 2;
  __syncthreads();
  for (int h = 1, lh = 0; h < P; h <<= 1, ++lh) {
    const int stride = ts * (N / (2 * h));
    for (int b = threadIdx.x; b < nseq * R * half; b += blockDim.x) {
      const int seq = b / half, bb = b - seq * half, j = bb & (h - 1);
      double2* p = z + (size_t)seq * P + ((bb >> lh) << (lh + 1)) + j;
      const double2 u = p[0], v = p[h];
      double2 w = v;
      if (h > 1) {
        const double c = cs[j * stride], s = sign * sn[j * stride];
        w = make_double2(fma(v.x, c, -v.y * s), fma(v.x, s, v.y * c));
      }
      p[0] = make_double2(u.x + w.x, u.y + w.y);
      p[h] = make_double2(u.x - w.x, u.y - w.y);
    }
    __syncthreads();
  }
  if (R == 1) return;
  const double s3 = sign * 0.86602540378443864676;  // exp(sign 2 pi i / 3) = -1/2 + i s3
  for (int b = threadIdx.x; b < nseq * P; b += blockDim.x) {
    const int seq = b / P, k = b - seq * P;
    double2* p = z + (size_t)seq * N + k;
    const double2 x0 = p[0], a = p[P], c = p[2 * P];
    const double c1 = cs[ts * k], s1 = sign * sn[ts * k], c2 = cs[2 * ts * k], s2 = sign * sn[2 * ts * k];
    const double2 y1 = make_double2(fma(a.x, c1, -a.y * s1), fma(a.x, s1, a.y * c1));
    const double2 y2 = make_double2(fma(c.x, c2, -c.y * s2), fma(c.x, s2, c.y * c2));
    const double sr = y1.x + y2.x, si = y1.y + y2.y, dr = s3 * (y1.x - y2.x), di = s3 * (y1.y - y2.y);
    const double hr = fma(-0.5, sr, x0.x), hi = fma(-0.5, si, x0.y);
    p[0] = make_double2(x0.x + sr, x0.y + si);
    p[P] = make_double2(hr - di, hi + dr);
    p[2 * P] = make_double2(hr + di, hi - dr);
  }
  __syncthreads();
}

// place of element q of a sequence of length N = R P before the passes
__device__ __forceinline__ int seq_place(int q, int R, int P, int bits) {
  const int rr = R == 3 ? q % 3 : 0, mm = R == 3 ? q / 3 : q;
  return rr * P + ves_bitrev(mm, bits);
}

__global__ void __launch_bounds__(256) interp_rows_kernel(int N, int Nup, int rows, int pairs,
                                                          const double* __restrict__ cs,
                                                          const double* __restrict__ sn,
                                                          const double* __restrict__ in, double scale,
                                                          double* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char interp_sm[];
  double2* z = reinterpret_cast<double2*>(interp_sm);  // [pairs][m][N]
  double2* y = z + (size_t)pairs * Nup;                // [pairs][N]
  const int m = Nup / N, R = (N % 3 == 0) ? 3 : 1, P = N / R, bits = __ffs(P) - 1;
  const long long b = blockIdx.y;
  const int row0 = blockIdx.x * 2 * pairs;
  const double* g = in + (b * rows + row0) * Nup;
  for (int pr = 0; pr < pairs; ++pr) {
    const bool on0 = row0 + 2 * pr < rows, on1 = row0 + 2 * pr + 1 < rows;
    const double* g0 = g + (long long)(2 * pr) * Nup;
    for (int c = threadIdx.x; c < Nup; c += blockDim.x) {
      const int q = c / m, r = c - q * m;
      z[((size_t)pr * m + r) * N + seq_place(q, R, P, bits)] = make_double2(on0 ? g0[c] : 0.0, on1 ? g0[Nup + c] : 0.0);
    }
  }
  seq_fft(z, pairs * m, N, cs, sn, 1.0, m);
  for (int i = threadIdx.x; i < pairs * N; i += blockDim.x) {
    const int pr = i / N, kk = i - pr * N;
    const double2* zk = z + (size_t)pr * Nup + kk;
    double ar = 0.0, ai = 0.0;
    if (2 * kk == N) {  // +-N/2, averaged: the real part of the twiddle
      for (int r = 0; r < m; ++r) {
        const double c = cs[(N / 2) * r];
        ar = fma(zk[(size_t)r * N].x, c, ar);
        ai = fma(zk[(size_t)r * N].y, c, ai);
      }
    } else {
      const int k = 2 * kk < N ? kk : kk - N, dk = k < 0 ? k + Nup : k;
      int t = 0;  // k r mod Nup
      for (int r = 0; r < m; ++r) {
        const double2 v = zk[(size_t)r * N];
        const double c = cs[t], s = sn[t];
        ar = fma(v.x, c, fma(-v.y, s, ar));
        ai = fma(v.x, s, fma(v.y, c, ai));
        t += dk;
        if (t >= Nup) t -= Nup;
      }
    }
    y[(size_t)pr * N + seq_place(kk, R, P, bits)] = make_double2(ar, ai);
  }
  seq_fft(y, pairs, N, cs, sn, -1.0, m);
  const double sc = scale / N;
  for (int i = threadIdx.x; i < pairs * N * 2; i += blockDim.x) {
    const int rr = i % (2 * pairs), k = i / (2 * pairs);
    if (row0 + rr >= rows) continue;
    const double2 v = y[(size_t)(rr >> 1) * N + k];
    out[(b * N + k) * rows + row0 + rr] = ((rr & 1) ? v.y : v.x) * sc;
  }
}

// Row pairs per CTA of the transform products: four, or as many as 96 KB of
// shared memory hold; 0: the sizes do not transform (N neither a power of two
// nor three times one, or one pair too large) and the dense products serve.
static int interp_pairs(int N, int Nup) {
  if (N % 2 || !ves_fft_size_ok(N)) return 0;
  const size_t per = (size_t)(Nup + N) * sizeof(double2);
  return (int)std::min<size_t>(4, 96 * 1024 / per);
}

// out[b] = scale * (in[b] P)^T for ``batch`` matrices of ``rows`` rows
static void launch_interp_rows(const ves_ctx* c, int pairs, int batch, int rows, const double* in, double scale,
                               double* out, cudaStream_t s) {
  const int N = c->N, Nup = c->Nup;
  const size_t sh = (size_t)pairs * (Nup + N) * sizeof(double2);
  if (sh > 48 * 1024) cudaFuncSetAttribute(interp_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
  for (int b0 = 0; b0 < batch; b0 += 65535) {
    const int nb = std::min(65535, batch - b0);
    ves_count_launch();
    interp_rows_kernel<<<dim3(ceil_div(rows, 2 * pairs), nb), 256, sh, s>>>(
        N, Nup, rows, pairs, c->cosU, c->sinU, in + (long long)b0 * rows * Nup, scale, out + (long long)b0 * rows * N);
  }
}

template <typename T>
__global__ void alpert_assemble_kernel(int N, const T* __restrict__ Gf, double* __restrict__ G, int k0) {
  const int kl = blockIdx.y;
  const long long NN = (long long)N * N;
  const T* g11 = Gf + (long long)kl * 3 * NN;
  const T* g12 = g11 + NN;
  const T* g22 = g12 + NN;
  double* Gk = G + (long long)(k0 + kl) * 4 * NN;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < 4 * NN; idx += gridDim.x * blockDim.x) {
    const int r = idx / (2 * N), c = idx % (2 * N);
    const int i = r % N, j = c % N;
    const T* src = (r < N) ? ((c < N) ? g11 : g12) : ((c < N) ? g12 : g22);
    Gk[idx] = (double)src[(long long)i * N + j];
  }
}

__global__ void nonfinite_check_kernel(long long n, const double* __restrict__ a, VesDeviceStatus* st) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    if (!isfinite(a[i])) {
      ves_set_error(st, VES_ERR_NONFINITE, 2, i);
      return;
    }
}

static int alpert_chunk(const ves_ctx* c, int nv, int precision) {
  const size_t es = precision == VES_PREC_FP64 ? 8 : 4;
  const size_t per = (size_t)3 * c->Nup * c->Nup * es;
  size_t budget = (size_t)2 << 30;  // ~2 GiB of Gup per chunk
  int ch = (int)(budget / per);
  if (ch < 1) ch = 1;
  if (ch > nv) ch = nv;
  return ch;
}

template <typename T>
static int alpert_impl(ves_ctx* c, int nv, const double* X, double* G, WsCarver& ws, cudaStream_t s) {
  const int N = c->N, Nup = c->Nup;
  const int chunk = alpert_chunk(c, nv, sizeof(T) == 8 ? VES_PREC_FP64 : VES_PREC_FP32C);
  double* Xup = ws.take<double>((size_t)nv * 2 * Nup);
  double* sa_up = ws.take<double>((size_t)nv * Nup);
  T* Fd = ws.take<T>((size_t)nv * Nup * 56);
  T* Gup = ws.take<T>((size_t)chunk * 3 * Nup * Nup);
  T* Tm = ws.take<T>((size_t)chunk * 3 * Nup * N);
  T* Gf = ws.take<T>((size_t)chunk * 3 * N * N);
  if (ws.sizing) return VES_OK;
  if (!ws.ok()) {
    ves_record_error(VES_ERR_WORKSPACE, "stokes_sl_matrix: workspace too small");
    return VES_ERR_WORKSPACE;
  }
  if (nv <= 0) return VES_OK;
  launch_upsample_deriv(c, nv, X, Xup, nullptr, sa_up, s);
  {
    dim3 grid(ceil_div(Nup, 128), nv);
    ves_count_launch();
    alpert_dense_nodes_kernel<T><<<grid, 128, (size_t)2 * N * sizeof(double), s>>>(N, Nup, c->m, c->nquad, X,
                                                                                   Xup, c->cq, c->qw, Fd);
  }
  const T* adense = (const T*)(sizeof(T) == 8 ? (const void*)c->adense : (const void*)c->adense32);
  const T* Pm = (const T*)(sizeof(T) == 8 ? (const void*)c->Pm : (const void*)c->Pm32);
  const T* Rm = (const T*)(sizeof(T) == 8 ? (const void*)c->Rm : (const void*)c->Rm32);
  constexpr int ROWS = 8;
  for (int k0 = 0; k0 < nv; k0 += chunk) {
    const int nk = min(chunk, nv - k0);
    dim3 grid(ceil_div(Nup, ROWS), nk);
    ves_count_launch();
    if (sizeof(T) == 4)
      alpert_rows_kernel<T, ROWS, 128, 9>
          <<<grid, 128, Nup * sizeof(float), s>>>(Nup, c->nquad, Xup, sa_up, adense, c->qw, Fd, Gup, k0);
    else
      alpert_rows_kernel<T, ROWS, 256, 1><<<grid, 256, 0, s>>>(Nup, c->nquad, Xup, sa_up, adense, c->qw, Fd, Gup, k0);
    const long long NN = (long long)Nup * Nup;
    // T = Gup * P for the 3*nk fields; Gf = R * T
    const int pairs = sizeof(T) == 8 ? interp_pairs(N, Nup) : 0;
    if (pairs > 0) {
      launch_interp_rows(c, pairs, 3 * nk, Nup, (const double*)Gup, 1.0, (double*)Tm, s);
      launch_interp_rows(c, pairs, 3 * nk, N, (const double*)Tm, (double)N / Nup, (double*)Gf, s);
    } else if (sizeof(T) == 8) {
      launch_bgemm_f64(3 * nk, Nup, N, Nup, 1.0, (const double*)Gup, Nup, NN, (const double*)Pm, N, 0, 0.0,
                       (double*)Tm, N, (long long)Nup * N, s);
      launch_bgemm_f64(3 * nk, N, N, Nup, 1.0, (const double*)Rm, Nup, 0, (const double*)Tm, N,
                       (long long)Nup * N, 0.0, (double*)Gf, N, (long long)N * N, s);
    } else {
      launch_bgemm_f32(3 * nk, Nup, N, Nup, 1.0f, (const float*)Gup, Nup, NN, (const float*)Pm, N, 0, 0.0f,
                       (float*)Tm, N, (long long)Nup * N, s);
      launch_bgemm_f32(3 * nk, N, N, Nup, 1.0f, (const float*)Rm, Nup, 0, (const float*)Tm, N,
                       (long long)Nup * N, 0.0f, (float*)Gf, N, (long long)N * N, s);
    }
    dim3 ga(ceil_div(4LL * N * N, 256), nk);
    ves_count_launch();
    alpert_assemble_kernel<T><<<ga, 256, 0, s>>>(N, Gf, G, k0);
  }
  ves_count_launch();
  nonfinite_check_kernel<<<256, 256, 0, s>>>((long long)nv * 4 * N * N, G, c->status);
  return ves_launch_check("stokes_sl_matrix");
}

int alpert_sl_matrix(ves_ctx* c, int nv, const double* X, int precision, double* G, WsCarver& ws,
                     cudaStream_t s) {
  if (precision == VES_PREC_FP64) return alpert_impl<double>(c, nv, X, G, ws, s);
  if (precision == VES_PREC_FP32C) return alpert_impl<float>(c, nv, X, G, ws, s);
  ves_record_error(VES_ERR_ARG, "stokes_sl_matrix: bad precision %d", precision);
  return VES_ERR_ARG;
}
