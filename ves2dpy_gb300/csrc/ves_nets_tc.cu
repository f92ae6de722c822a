// Tensor-core (tcgen05, BF16 operands, FP32 accumulation) path of the MLARM
// network engine.  Same block template as ves_nets.cu; every convolution is a
// sum of shifted GEMMs
//     D[o][p] += sum_c W_s[o][c] * X[p + s][c]
// with D (positions x output channels) in tensor memory, X (positions x
// channels, the MMA's A operand) and W_s (output channels x channels, one
// matrix per input shift s, the B operand) K-major in shared memory.  A shift
// is a start-address offset of X's descriptor (ves_tc.cuh), so no im2col copy
// is made:
//   * stride-2 convolutions read the input split by position parity, with
//     circular halos of 3 rows: input position 2p + s is row p + (s >> 1) of
//     parity s & 1; the two branches (dilation 1 and 2) share the shifts
//     -6..6 (except +-5) and fill the output rows [0, c1) and [c1, 2c1);
//   * transposed convolutions (kernel 10, stride 2, padding 4) are split by
//     output parity r: out[2q + r] = sum_{u<5} W[r + 2u] in[q + 2 - u], zero
//     halos of 2 rows;
//   * the mixing convolution (kernel 3) reads shifts -1, 0, 1 of a zero-halo
//     array.
// Positions are the MMA's M = 128 rows (one TMEM lane each, so every thread of
// an epilogue owns one position and writes 16-byte rows of 8 channels);
// layers with fewer positions leave the remaining rows to read whatever
// follows in shared memory, and those rows are never read back.  Output
// channels are N, rounded up to 16.
//
// Three kernels per block: "down" (conv pair 1, conv pair 2), "up1"
// (transposed conv 1) and "up2" (transposed conv 2, mix, residual and
// pass-through).  All work on tiles of V vesicles of one group whose rows are
// interleaved (row q*V + j holds position q of the tile's vesicle j), so that
// the MMAs use all 128 rows: a shift of the input by u positions is a shift
// by u*V rows, and every row still only meets rows of its own vesicle.  down:
// two vesicles at L = 128 (conv pair 1 fills 128 rows, conv pair 2 64), one at
// L = 256; up1: 128 / (L/4); up2: two at L = 128, one at L = 256.  down and
// up1 write the intermediate in the next kernel's layout.  The block input and
// output stay FP32 in global memory ([nv][groups*channels][L]); the
// intermediates between the kernels are BF16 in the K-major layout.  Kernels
// are persistent: each CTA walks a contiguous range of (group, tile) items,
// loading a group's weight image into shared memory once per group it meets,
// and runs two or three warp groups of eight warps (as TMEM and shared memory
// allow), each on its own items: while one waits for its MMAs the others run
// their epilogues.
//
// What bounds them, from clock stamps in a copy: the tensor core's reads of its
// operands from shared memory (an M = 128, N = 128, K = 16 MMA reads 8 KB in
// its 64 cycles, the whole shared-memory rate) next to the epilogues' own
// reads and writes there.  With every epilogue access left out of the copy
// the kernels still took 75-95% of their time.  One network pass, 1024
// vesicles, ms: advection 56.1 -> 49.3, near field 48.7 -> 34.9,
// advection-tension 42.5 -> 31.8.  The near field's kernels: down 1.20 -> 0.92, up1 0.45 -> 0.33,
// up2 1.83 -> 1.23; the advection's 1.67 -> 1.41, 0.62 -> 0.51, 2.05 -> 1.86.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "ves_internal.h"
#include "ves_tc.cuh"
#include <cuda_bf16.h>

namespace tcnet {

constexpr int kGroupThreads = 256;  // eight warps: two on each TMEM lane quarter
constexpr int kMinSmem = 117 * 1024;
constexpr int kOffsets = 11;  // input shifts of a conv pair: -6..6 without +-5
__host__ __device__ constexpr int shift_of(int oi) { return oi < 2 ? -6 + 2 * oi : (oi < 9 ? oi - 5 : 2 * oi - 14); }

__host__ __device__ constexpr int rup(int a, int b) { return (a + b - 1) / b * b; }

// Geometry of one block, shared by host packing and kernels (bytes unless noted).
// Shared memory holds one weight image and, per warp group, its own
// activation arrays (each warp group runs its own (group, vesicle) items).
struct Geo {
  int cin, c1, c2, cmix, residual, npass, L, lgL;
  int n1, d;             // conv-pair output channels
  int kcin, kc1, kcd;    // 8-channel K chunks of the three GEMM inputs (even)
  // down image: W1 [11][kcin][n1][16B], W2 [11][kc1][d][16B], consts [6][128] f32
  int dw1, dw2, dcst, dsize;
  // down arrays of warp group 0 (group k at + k*dgrp): xs [2][kcin][L/2+6][16B],
  // as [2][kc1][L/4+6][16B], xf [cin][L] f32 (the
  // block input as it arrives by bulk copy); a tail of 2 KB follows the groups
  int dxs, das, dxf, dgrp;
  // up1 image (transposed conv 1): W (u1merge = 0: [2][5][kcd][d][16B], output
  // parity r, tap u, the parities M-split over the lanes; u1merge = 1: the
  // merged layout of up2, both parities in one operand of N = 2*kcd*8),
  // consts [7][128] f32; arrays of warp group 0: bs [kcd][L/4+4][16B]
  int u1merge, u1w, u1cst, u1size, u1bs, u1grp;
  // up2 image (transposed conv 2 and mix): W (u2merge = 1: [5][kcd][2*kcd*8][16B],
  // both output parities in one operand of N = 2*kcd*8 rows, parity r at row
  // r*kcd*8; u2merge = 0: as up1), M [3][kcd][cmix][16B], consts [7][128] f32;
  // arrays of warp group 0: cs [kcd][(L/2+4)*vu][16B], ds [kcd][(L+2)*vu][16B]
  int u2merge, u2w, u2wm, u2cst, u2size, u2cs, u2ds, u2grp;
  // down -> up1 per tile of v1 vesicles: [kcd][L/4][v1][16B] (mid_bytes per
  // vesicle); up1 -> up2 per tile of vu vesicles: [kcd][L/2][vu][16B]
  int mid_bytes, mid2_bytes, mid_stride;
  int v1;  // vesicles per up1 tile (v1 * L/4 = 128 rows)
  int vu;  // vesicles per up2 tile (2 at L = 128 when two tiles fit on an SM)
  int vd;  // vesicles per down tile (2 at L = 128: the block input is read
           // from global memory (L2-prefetched) with no FP32 staging copy)
};

constexpr int kMaxSmem = 227 * 1024 - 256;  // dynamic shared memory available next to the static part
constexpr int kTail = 128 * 16;             // after the groups' arrays: rows an MMA reads past the last one

// byte offset of row o of K chunk kc of tap u, output parity r, in the
// unmerged layout [2][5][kcd][d][16B] (base = start of the weights)
__host__ __device__ inline int dec_w_off(const Geo& g, int base, int r, int u, int kc, int o) {
  return base + (((r * 5 + u) * g.kcd + kc) * g.d + o) * 16;
}
// same in the merged layout [5][kcd][2*kcd*8][16B]
__host__ __device__ inline int dec_w_off_merged(const Geo& g, int base, int r, int u, int kc, int o) {
  return base + ((u * g.kcd + kc) * 2 * g.kcd * 8 + r * g.kcd * 8 + o) * 16;
}

// transposed conv 1 with both output parities in one MMA (VES_TC_UP1_MERGE=0/1
// overrides the default; read once)
inline int tcnet_up1_merge(int L) {
  static int v = -2;
  if (v == -2) {
    const char* e = getenv("VES_TC_UP1_MERGE");
    v = e ? (atoi(e) ? 1 : 0) : -1;
  }
  if (v >= 0) return v;
  (void)L;
  return 1;  // measured 1-2% faster networks than the M-split at L = 128 and 256
}

inline Geo make_geo(const ves_net_block& b, int L) {
  Geo g;
  g.cin = b.cin;
  g.c1 = b.c1;
  g.c2 = b.c2;
  g.cmix = b.cmix;
  g.residual = b.residual;
  g.npass = b.npass;
  g.L = L;
  g.lgL = 0;
  while ((1 << g.lgL) < L) ++g.lgL;
  g.n1 = 2 * b.c1;
  g.d = 2 * b.c2;
  g.kcin = rup(b.cin, 16) / 8;
  g.kc1 = rup(g.n1, 16) / 8;
  g.kcd = rup(g.d, 16) / 8;
  int o = 0;
  g.dw1 = o;
  o += kOffsets * g.kcin * g.n1 * 16;
  g.dw2 = o;
  o += kOffsets * g.kc1 * g.d * 16;
  g.dcst = o;
  o += 6 * 128 * 4;
  g.dsize = o;
  g.vd = (L / 2 <= 64) ? 2 : 1;
  g.dxs = o;
  o += 2 * g.kcin * (L / 2 + 6) * g.vd * 16;
  g.das = o;
  o += 2 * g.kc1 * (L / 4 + 6) * g.vd * 16;
  g.dxf = o;
  o += g.vd == 1 ? rup(g.cin * L * 4, 16) : 0;
  g.dgrp = o - g.dxs;
  const int dec_unmerged = 10 * g.kcd * g.d * 16;
  // up1: both parities in one MMA of N = 2*Nd (u1merge, fewer and larger MMAs,
  // half the lanes busy) or M-split over the lanes (unmerged layout)
  g.u1merge = tcnet_up1_merge(L);
  g.u1w = 0;
  g.u1cst = g.u1merge ? 5 * g.kcd * 2 * g.kcd * 8 * 16 : dec_unmerged;
  g.u1size = g.u1cst + 7 * 128 * 4;
  g.u1bs = g.u1size;
  g.v1 = 128 / (L / 4);
  g.u1grp = g.kcd * (L / 4 + 4) * g.v1 * 16;
  // up2: tiles of two vesicles at L = 128 (128 rows) when two warp groups of
  // them fit in shared memory and TMEM; merged image (both parities in one
  // operand of N = 2*Nd rows) when two groups fit next to it
  auto lay_up2 = [&](int vu, int merge) {
    g.vu = vu;
    g.u2merge = merge;
    g.u2w = 0;
    g.u2wm = merge ? 5 * g.kcd * 2 * g.kcd * 8 * 16 : dec_unmerged;
    g.u2cst = g.u2wm + 3 * g.kcd * g.cmix * 16;
    g.u2size = g.u2cst + 7 * 128 * 4;
    g.u2grp = g.kcd * (L / 2 + 4 + L + 2) * vu * 16;
    return g.u2size + 2 * g.u2grp + kTail <= kMaxSmem;
  };
  if (!(L == 128 && 2 * (2 * g.kcd * 8 + 64) <= 512 && lay_up2(2, 1)) && !lay_up2(1, 1)) lay_up2(1, 0);
  g.u2cs = g.u2size;
  g.u2ds = g.u2cs + g.kcd * (L / 2 + 4) * g.vu * 16;
  g.mid_bytes = g.kcd * (L / 4) * 16;
  g.mid2_bytes = g.kcd * (L / 2) * 16;
  g.mid_stride = g.mid_bytes + g.mid2_bytes;
  return g;
}

struct KArgs {
  Geo g;
  int G, nv;
  long long items;
  const unsigned char* img;  // group 0 image of this block; group stride = image size
  const float* x;            // block input [nv][G*cin][L]
  float* out;                // block output [nv][G*cout][L]
  unsigned char* mid;        // down -> up1: [ntiles][G][v1 * mid_bytes]
  unsigned char* mid2;       // up1 -> up2: [tiles of vu][G][vu * mid2_bytes]
  int per_grp;               // items per channel group (tiles of the kernel's vesicles)
  VesDeviceStatus* st;
};

__device__ __forceinline__ void copy16(unsigned char* dst, const unsigned char* src, int bytes) {
  const uint4* s = reinterpret_cast<const uint4*>(src);
  uint4* d = reinterpret_cast<uint4*>(dst);
  for (int i = threadIdx.x; i < bytes / 16; i += blockDim.x) d[i] = s[i];
}
__device__ __forceinline__ void zero16(unsigned char* dst, int bytes) {
  uint4* d = reinterpret_cast<uint4*>(dst);
  const uint4 z = make_uint4(0, 0, 0, 0);
  for (int i = threadIdx.x; i < bytes / 16; i += blockDim.x) d[i] = z;
}

// barrier of one warp group (named barrier 1 + group)
__device__ __forceinline__ void group_sync(int wg) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + wg), "r"(kGroupThreads) : "memory");
}
// all of the group's writes to shared memory so far -> visible to the tensor core
__device__ __forceinline__ void group_sync_for_mma(int wg) {
  tc_fence_async_smem();
  tc_fence_before_sync();
  group_sync(wg);
  tc_fence_after_sync();
}
// Bounded wait of one warp group on an mbarrier; true when the phase
// completed (the answer is uniform across the group).  Thread 0 of the group
// polls (sleeping between polls) and the others wait in the group barrier, so
// a wait that is not yet satisfied takes no issue slots from the other groups.
__device__ __forceinline__ bool group_wait_one(uint64_t* bar, unsigned phase, VesDeviceStatus* st, int site, int wg,
                                               int gt, int* flag) {
  if (gt == 0 && !tc_mbar_wait_sleep(bar, phase, st, site)) atomicExch(flag, 1);
  group_sync(wg);
  return *(volatile int*)flag == 0;
}

// The tensor core takes MMAs in the order they are issued.  Groups that issue
// at the same time share its rate, finish together and then all run their
// epilogues while it idles; a group that issues its whole batch before the
// next one starts leaves the others' epilogues to overlap with it.  The
// issuing threads therefore take turns through a flag in shared memory.  It
// orders issue only: one that waits too long issues anyway.
__device__ __forceinline__ void batch_begin(int* flag) {
  for (int it = 0; it < (1 << 14); ++it)
    if (*(volatile int*)flag == 0 && atomicCAS(flag, 0, 1) == 0) return;
}
__device__ __forceinline__ void batch_end(int* flag) { atomicExch(flag, 0); }

// MMA issue sequences.  One elected thread of a group's first warp issues;
// the operands are computed from values that are the same across the warp
// (the group's index and the TMEM base by a shuffle, everything else from
// kernel arguments), which lets descriptors stay in uniform registers: from
// per-thread values an issue took 65-75 cycles whatever the shape, like this
// 37-51 where the tensor core takes 32-44.  The issuing lane runs the
// sequences as straight-line code:
// each is a template on the number of 16-channel K steps (NK), picked by one
// switch, so that no loop branch sits between two tcgen05.mma (a branching
// loop in the single issuing lane costs more than the tensor core's time per
// MMA).  Descriptors advance by adds: the start address is the low 14 bits of
// a descriptor, in 16-byte units.

// conv pair: 11 input shifts x NK K steps.  A at a0 + par*aPar + row*rowMul
// (rowMul: vesicles per tile, rows interleaved), B at b0 + oi*bOi; K steps at
// stepA / stepB.
template <int NK>
__device__ __forceinline__ void issue_conv(uint32_t d, uint64_t a0, uint64_t b0, uint32_t aPar, uint32_t bOi,
                                           uint32_t stepA, uint32_t stepB, uint32_t idesc, uint32_t rowMul = 1) {
#pragma unroll
  for (int oi = 0; oi < kOffsets; ++oi) {
    const int s = shift_of(oi);
    const uint64_t ad = a0 + (uint32_t)((s & 1) * aPar + (3 + (s >> 1)) * rowMul);
    const uint64_t bd = b0 + (uint32_t)oi * bOi;
#pragma unroll
    for (int j = 0; j < NK; ++j) tc_mma_bf16(d, ad + j * stepA, bd + j * stepB, idesc, (oi | j) ? 1u : 0u);
  }
}
// transposed conv, one output parity: 5 taps u (A rows (4 - u) * tapRows) x NK K steps.
template <int NK>
__device__ __forceinline__ void issue_deconv(uint32_t d, uint64_t a0, uint64_t b0, uint32_t bTap, uint32_t stepA,
                                             uint32_t stepB, uint32_t idesc, uint32_t tapRows = 1) {
#pragma unroll
  for (int u = 0; u < 5; ++u) {
    const uint64_t ad = a0 + (uint32_t)(4 - u) * tapRows, bd = b0 + (uint32_t)u * bTap;
#pragma unroll
    for (int j = 0; j < NK; ++j) tc_mma_bf16(d, ad + j * stepA, bd + j * stepB, idesc, (u | j) ? 1u : 0u);
  }
}
// mix of 128 rows: 3 taps t (A rows t * tapRows) x NK K steps, onto the
// preset accumulator
template <int NK>
__device__ __forceinline__ void issue_mix(uint32_t d, uint64_t a0, uint64_t b0, uint32_t bTap, uint32_t stepA,
                                          uint32_t stepB, uint32_t idesc, uint32_t tapRows) {
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const uint64_t ad = a0 + (uint32_t)t * tapRows, bd = b0 + (uint32_t)t * bTap;
#pragma unroll
    for (int j = 0; j < NK; ++j) tc_mma_bf16(d, ad + j * stepA, bd + j * stepB, idesc, 1u);
  }
}
#define VES_TC_NK_SWITCH(nk, call)                                                                            \
  switch (nk) {                                                                                               \
    case 1: call(1); break;                                                                                   \
    case 2: call(2); break;                                                                                   \
    case 3: call(3); break;                                                                                   \
    case 4: call(4); break;                                                                                   \
    case 5: call(5); break;                                                                                   \
    case 6: call(6); break;                                                                                   \
    case 7: call(7); break;                                                                                   \
    default: call(8); break;                                                                                  \
  }

struct Range {
  long long lo, hi;
};
__device__ __forceinline__ Range my_items(long long items) {
  const long long per = items / gridDim.x, rem = items % gridDim.x;
  const long long b = blockIdx.x;
  const long long lo = b * per + (b < rem ? b : rem);
  return {lo, lo + per + (b < rem ? 1 : 0)};
}

// ---------------------------------------------------------------------------
// Epilogue helpers.  D[p][c] sits in TMEM with the position p on lane p and
// the channel c in column c; each thread owns one position and reads 8
// channels at a time, which is one 16-byte row of the next layer's K-major
// operand.

// two FP32 values -> one 32-bit word of two BF16 (round to nearest even), low half first
__device__ __forceinline__ uint32_t pack_bf2(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// 8 channels [8kc, 8kc+8) of this thread's position: relu(v + b) * s + t, 0 beyond nreal
__device__ __forceinline__ uint4 act8(const float* v, const float* cst, int kc, int nreal, int ob, int os, int ot) {
  float b[8], sc[8], sh[8];
  *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(cst + ob + 8 * kc);
  *reinterpret_cast<float4*>(b + 4) = *reinterpret_cast<const float4*>(cst + ob + 8 * kc + 4);
  *reinterpret_cast<float4*>(sc) = *reinterpret_cast<const float4*>(cst + os + 8 * kc);
  *reinterpret_cast<float4*>(sc + 4) = *reinterpret_cast<const float4*>(cst + os + 8 * kc + 4);
  *reinterpret_cast<float4*>(sh) = *reinterpret_cast<const float4*>(cst + ot + 8 * kc);
  *reinterpret_cast<float4*>(sh + 4) = *reinterpret_cast<const float4*>(cst + ot + 8 * kc + 4);
  float y[8];
  // packed FP32x2 add and fma: per lane the same rounding as fadd / fmaf
#pragma unroll
  for (int e = 0; e < 8; e += 2) {
    float2 z = __fadd2_rn(make_float2(v[e], v[e + 1]), make_float2(b[e], b[e + 1]));
    z.x = fmaxf(z.x, 0.f);
    z.y = fmaxf(z.y, 0.f);
    z = __ffma2_rn(z, make_float2(sc[e], sc[e + 1]), make_float2(sh[e], sh[e + 1]));
    y[e] = z.x;
    y[e + 1] = z.y;
  }
  if (8 * kc + 8 > nreal) {  // the chunk that holds the padding channels (TMEM columns past nreal are not defined)
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (8 * kc + e >= nreal) y[e] = 0.f;
  }
  return make_uint4(pack_bf2(y[0], y[1]), pack_bf2(y[2], y[3]), pack_bf2(y[4], y[5]), pack_bf2(y[6], y[7]));
}

// ---------------------------------------------------------------------------
// Segments: the CTA's contiguous item range split where the channel group
// changes; the weight image is reloaded (whole CTA) at each segment start and
// the warp groups take the segment's items in turn.
struct Seg {
  long long lo, hi;
  int grp;
};
__device__ __forceinline__ Seg next_seg(long long lo, long long hi, int nv) {
  const int grp = (int)(lo / nv);
  const long long end = (long long)(grp + 1) * nv;
  return {lo, end < hi ? end : hi, grp};
}

// down: conv pairs 1 and 2 on tiles of VD vesicles with interleaved rows (128
// rows of conv pair 1, 64 of conv pair 2).  KC1 / KCD: compile-time K chunk
// counts of the two conv pairs' outputs (0: read them from the geometry), so
// that every epilogue and issue loop unrolls.  NG warp groups of eight warps,
// each running its own tiles (2: 256 TMEM columns each; 3: 128, when N1 + N2
// <= 128 and the groups' arrays fit in shared memory).
template <int KC1, int KCD, int NG, int VD>
__global__ void __launch_bounds__(NG * kGroupThreads, 1) down_kernel(KArgs a) {
  extern __shared__ __align__(128) unsigned char sm[];
  __shared__ uint64_t bar[NG], xbar[NG];  // per warp group: MMA completion, input arrival
  __shared__ uint32_t tbase;
  __shared__ int fail[NG];
  const Geo& g = a.g;
  const int kc1 = KC1 ? KC1 : g.kc1, kcd = KCD ? KCD : g.kcd;
  const int L = g.L, L2 = L / 2, L4 = L / 4;
  const int ntl = a.per_grp;    // tiles per channel group
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wg = tid / kGroupThreads, gt = tid % kGroupThreads;    // warp group, thread within it
  const int qd = warp & 3, hw = gt >> 7;   // TMEM lane quarter; which of the two warps on it
  const Range rg = my_items(a.items);
  if (rg.lo >= rg.hi) return;
  const uint32_t ncols = 512;  // all of TMEM (one CTA per SM)
  if (tid == 0) {
    for (int k = 0; k < NG; ++k) {
      tc_mbar_init(&bar[k], 1);
      tc_mbar_init(&xbar[k], 1);
      fail[k] = 0;
    }
    tc_mbar_fence_init();
  }
  if (warp == 0) tc_tmem_alloc(&tbase, ncols);
  zero16(sm + g.dxs, NG * g.dgrp + 128 * 16);  // K padding of the activation arrays stays zero
  tc_fence_async_smem();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const int N1 = kc1 * 8, N2 = kcd * 8;
  const int wgu = __shfl_sync(0xffffffffu, wg, 0);  // uniform across the warp
  const bool issuer = __shfl_sync(0xffffffffu, gt >> 5, 0) == 0 && tc_elect();
  const uint32_t tcol = __shfl_sync(0xffffffffu, tbase, 0) + (NG == 2 ? 256 : 128) * wgu;
  const uint32_t d1 = tcol, d2 = tcol + N1;
  const uint32_t lanes = (uint32_t)(32 * qd) << 16;
  const uint32_t sbase = tc_smem_u32(sm);
  const int goff = wgu * g.dgrp;
  const float* cst = reinterpret_cast<const float*>(sm + g.dcst);
  const int P1 = (L2 + 6) * VD, P2 = (L4 + 6) * VD;  // rows per K chunk (circular halos of 3 positions)
  uint4* xs = reinterpret_cast<uint4*>(sm + g.dxs + goff);
  uint4* as = reinterpret_cast<uint4*>(sm + g.das + goff);
  float* xf = reinterpret_cast<float*>(sm + g.dxf + goff);
  const uint32_t xbytes = (uint32_t)(g.cin * L * 4);
  unsigned phase = 0, xphase = 0;
  bool xpend = false;  // a bulk copy into xf is in flight
  // block input x[v][grp*cin + c][pos] (cin*L contiguous floats) of a tile's
  // vesicles: one vesicle -> xf by bulk copy; a tile of two -> L2
  // (read by convert_x straight from global memory)
  auto fetch_x = [&](int grp, long long t) {
    if (VD == 1) {
      if (gt == 0) {
        tc_expect_tx(&xbar[wg], xbytes);
        tc_bulk_g2s(xf, a.x + (t * a.G + grp) * (long long)g.cin * L, xbytes, &xbar[wg]);
      }
      xpend = true;
    } else if (gt < VD && t * VD + gt < a.nv) {
      tc_prefetch_l2(a.x + ((t * VD + gt) * a.G + grp) * (long long)g.cin * L, xbytes);
    }
  };
  // block input -> parity-split BF16 rows with circular halos of 3
  // positions, position m of vesicle j at row (m + 3)*VD + j; one thread per
  // (8-channel chunk, vesicle, position pair 2m, 2m+1)
  auto convert_x = [&](long long t, int grp) {
    const int lg2 = g.lgL - 1;
#pragma unroll 2
    for (int i = gt; i < g.kcin * VD * L2; i += kGroupThreads) {
      const int m = i & (L2 - 1), kj = i >> lg2, kc = kj / VD, j = kj - kc * VD;
      const long long v = t * VD + j;
      float2 y[8];
      if (VD == 1) {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          y[e] = (8 * kc + e < g.cin) ? *reinterpret_cast<const float2*>(xf + (8 * kc + e) * L + 2 * m)
                                      : make_float2(0.f, 0.f);
      } else {
        const float* src = a.x + ((v < a.nv ? v : 0) * a.G + grp) * (long long)g.cin * L;
#pragma unroll
        for (int e = 0; e < 8; ++e)
          y[e] = (8 * kc + e < g.cin && v < a.nv) ? __ldg(reinterpret_cast<const float2*>(src + (8 * kc + e) * L + 2 * m))
                                                  : make_float2(0.f, 0.f);
      }
      const uint4 v0 = make_uint4(pack_bf2(y[0].x, y[1].x), pack_bf2(y[2].x, y[3].x), pack_bf2(y[4].x, y[5].x),
                                  pack_bf2(y[6].x, y[7].x));
      const uint4 v1 = make_uint4(pack_bf2(y[0].y, y[1].y), pack_bf2(y[2].y, y[3].y), pack_bf2(y[4].y, y[5].y),
                                  pack_bf2(y[6].y, y[7].y));
      uint4* b0 = xs + (size_t)kc * P1 + j;
      uint4* b1 = xs + (size_t)(g.kcin + kc) * P1 + j;
      b0[(m + 3) * VD] = v0;
      b1[(m + 3) * VD] = v1;
      if (m >= L2 - 3) {
        b0[(m + 3 - L2) * VD] = v0;
        b1[(m + 3 - L2) * VD] = v1;
      }
      if (m < 3) {
        b0[(m + 3 + L2) * VD] = v0;
        b1[(m + 3 + L2) * VD] = v1;
      }
    }
  };
  bool failed = false, stuck = false;  // stuck: this warp group's own MMA wait timed out
  for (long long lo = rg.lo; lo < rg.hi && !failed;) {
    const Seg sg = next_seg(lo, rg.hi, ntl);
    const long long t0 = (long long)sg.grp * ntl;  // first item of the group
    __syncthreads();
    copy16(sm, a.img + (size_t)sg.grp * g.dsize, g.dsize);  // whole CTA
    tc_fence_async_smem();  // weights (and the zeroed padding) -> tensor core, for every group
    __syncthreads();
    if (sg.lo + wg < sg.hi) fetch_x(sg.grp, sg.lo + wg - t0);
    for (long long it = sg.lo + wg; it < sg.hi; it += NG) {
      const long long t = it - t0;
      if (VD == 1) {
        if (!group_wait_one(&xbar[wg], xphase, a.st, 20, wg, gt, &fail[wg])) {
          failed = true;
          break;
        }
        xphase ^= 1;
        xpend = false;
      }
      convert_x(t, sg.grp);
      group_sync_for_mma(wg);  // xs complete; xf fully read
      // conv pair 1: D1[r][o], rows r = p*VD + j (p < L/2) on the lanes, o < n1 in the columns
      if (issuer) {
        const uint32_t idesc = tc_idesc_bf16(128, N1);
        const uint32_t lboA = P1 * 16, lboB = g.n1 * 16;
        const uint64_t a0 = tc_desc(sbase + g.dxs + goff, lboA, 128), b0 = tc_desc(sbase + g.dw1, lboB, 128);
#define VES_CONV1(NK) issue_conv<NK>(d1, a0, b0, (g.kcin * lboA) >> 4, (g.kcin * lboB) >> 4, (2 * lboA) >> 4, (2 * lboB) >> 4, idesc, (uint32_t)VD)
        VES_TC_NK_SWITCH(g.kcin / 2, VES_CONV1)
#undef VES_CONV1
        tc_commit(&bar[wgu]);
      }
      if (it + NG < sg.hi) fetch_x(sg.grp, t + NG);
      if (!group_wait_one(&bar[wg], phase, a.st, 21, wg, gt, &fail[wg])) {
        failed = stuck = true;
        break;
      }
      phase ^= 1;
      tc_fence_after_sync();
      // the epilogue's row r holds position p = r / VD of the tile's vesicle j = r % VD;
      // conv pair 2 reads position q of parity par at row (q + 3)*VD + j
      if (32 * qd < L2 * VD) {  // uniform per warp: the TMEM loads are warp-wide
        const int r = 32 * qd + lane, p = r / VD, j = r % VD, par = p & 1, q = p >> 1;
        const bool own = p < L2;
        const int k1 = hw ? kc1 : kc1 / 2;
#pragma unroll
        for (int kk = 0; kk < (KC1 ? KC1 / 2 : 8); kk += 4) {
          const int k0 = hw * (kc1 / 2) + kk;
          if (k0 >= k1) break;
          float vv[32];
          tc_ld32(d1 + lanes + 8 * k0, vv);
          if (own) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              if ((KC1 != 0 && kk + k >= KC1 / 2) || k0 + k >= k1) break;
              const uint4 val = act8(vv + 8 * k, cst, k0 + k, g.n1, 0, 128, 256);
              uint4* base = as + (size_t)(par * kc1 + k0 + k) * P2 + j;
              base[(q + 3) * VD] = val;
              if (q >= L4 - 3) base[(q + 3 - L4) * VD] = val;
              if (q < 3) base[(q + 3 + L4) * VD] = val;
            }
          }
        }
      }
      group_sync_for_mma(wg);
      // conv pair 2: D2[r][o], rows r = p*VD + j (p < L/4, 64 rows), o < d; M = 64
      // halves the operand read per MMA
      constexpr int M2 = KCD ? 64 : 128;
      if (issuer) {
        const uint32_t idesc = tc_idesc_bf16(M2, N2);
        const uint32_t lboA = P2 * 16, lboB = g.d * 16;
        const uint64_t a0 = tc_desc(sbase + g.das + goff, lboA, 128), b0 = tc_desc(sbase + g.dw2, lboB, 128);
#define VES_CONV2(NK) issue_conv<NK>(d2, a0, b0, (kc1 * lboA) >> 4, (kc1 * lboB) >> 4, (2 * lboA) >> 4, (2 * lboB) >> 4, idesc, (uint32_t)VD)
        VES_TC_NK_SWITCH(kc1 / 2, VES_CONV2)
#undef VES_CONV2
        tc_commit(&bar[wgu]);
      }
      if (!group_wait_one(&bar[wg], phase, a.st, 22, wg, gt, &fail[wg])) {
        failed = stuck = true;
        break;
      }
      phase ^= 1;
      tc_fence_after_sync();
      // the intermediate goes straight to global memory: row (kc, p) of
      // vesicle v = t*VD + j sits in its up1 tile (v / v1) at ((kc * L/4 + p) * v1 + v % v1)
      const int V1 = g.v1;
      if (KCD != 0) {
        // rows 16 qd .. + 15 of this quarter; the half-warps take the two
        // halves of the channel chunks (16x32bx2 loads), the two warps parts of each half
        const int r = 16 * qd + (lane & 15), p = r / VD, j = r % VD;
        const long long v = t * VD + j;
        const int kb = (lane >> 4) * (KCD / 2);
        const long long vs = v < a.nv ? v : 0;
        uint4* gmid = reinterpret_cast<uint4*>(a.mid + ((size_t)(vs / V1) * a.G + sg.grp) * (size_t)V1 * g.mid_bytes) +
                      (vs % V1);
        float vv[32];
        tc_ld16x2_32<4 * KCD>(d2 + lanes, vv);
        if (p < L4 && v < a.nv) {
#pragma unroll
          for (int k = 0; k < KCD / 2; ++k)
            if ((k < (KCD / 2 + 1) / 2) == (hw == 0))
              gmid[((size_t)(kb + k) * L4 + p) * V1] = act8(vv + 8 * k, cst, kb + k, g.d, 384, 512, 640);
        }
      } else if (32 * qd < L4 * VD) {
        const int r = 32 * qd + lane, p = r / VD, j = r % VD;
        const long long v = t * VD + j;
        const bool own = p < L4 && v < a.nv;
        const long long vs = own ? v : 0;
        uint4* gmid = reinterpret_cast<uint4*>(a.mid + ((size_t)(vs / V1) * a.G + sg.grp) * (size_t)V1 * g.mid_bytes) +
                      (vs % V1);
        const int k1 = hw ? kcd : kcd / 2;
#pragma unroll
        for (int kk = 0; kk < 8; kk += 4) {
          const int k0 = hw * (kcd / 2) + kk;
          if (k0 >= k1) break;
          float vv[32];
          tc_ld32(d2 + lanes + 8 * k0, vv);
          if (own) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (k0 + k < k1)
                gmid[((size_t)(k0 + k) * L4 + p) * V1] = act8(vv + 8 * k, cst, k0 + k, g.d, 384, 512, 640);
          }
        }
      }
      tc_fence_before_sync();
      group_sync(wg);  // every TMEM read done before the next item's MMAs
    }
    lo = sg.hi;
    failed = __syncthreads_or(failed ? 1 : 0) != 0;  // every thread takes part
  }
  // bounded drains: this group's MMAs and bulk copies still in flight after a failure
  if (stuck) tc_mbar_wait(&bar[wg], phase, nullptr, 0);
  if (xpend) tc_mbar_wait(&xbar[wg], xphase, nullptr, 0);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tc_tmem_dealloc(tbase, ncols);
}

// ---------------------------------------------------------------------------
// The transposed convolutions, split in two kernels so that their weight
// images and per-group arrays are small enough for several warp groups per SM:
//   up1: transposed conv 1 (intermediate [kcd][L/4] -> [kcd][L/2], BF16 rows
//        to global memory);
//   up2: transposed conv 2, mix, residual and pass-through channels.
// Both output parities share one MMA of N = 2*Nd (merged image) or run as two
// MMAs on the same lanes; parity r accumulates in TMEM columns [r*Nd, (r+1)*Nd)
// either way.

// Issue one transposed conv (thread 0 of the group).  w0/w1: byte offsets of
// parity 0/1 weights (tap 0, chunk 0, row 0), bTap: tap stride (16-byte
// units), lboB: K-chunk stride of B in bytes, merged: both parities in one
// operand of N = 2*Nd rows at w0; tapRows: vesicles per tile, rows interleaved.
template <int KCD>
__device__ __forceinline__ void deconv_issue(uint32_t dt, uint32_t sbase, uint32_t a_off, uint32_t lboA, int Nd,
                                             int kcd, bool merged, uint32_t w0, uint32_t w1, uint32_t bTap,
                                             uint32_t lboB, uint32_t tapRows) {
  const uint32_t stepA = (2 * lboA) >> 4;
  const uint64_t a0 = tc_desc(sbase + a_off, lboA, 128);
  if (merged) {
    const uint32_t idesc = tc_idesc_bf16(128, 2 * Nd);
    const uint64_t b0 = tc_desc(sbase + w0, lboB, 128);
#define VES_DEC(NK) issue_deconv<NK>(dt, a0, b0, bTap, stepA, (2 * lboB) >> 4, idesc, tapRows)
    VES_TC_NK_SWITCH(kcd / 2, VES_DEC)
#undef VES_DEC
  } else {
    const uint32_t idesc = tc_idesc_bf16(128, Nd);
    for (int r = 0; r < 2; ++r) {
      const uint64_t b0 = tc_desc(sbase + (r ? w1 : w0), lboB, 128);
#define VES_DEC(NK) issue_deconv<NK>(dt + r * Nd, a0, b0, bTap, stepA, (2 * lboB) >> 4, idesc, tapRows)
      VES_TC_NK_SWITCH(kcd / 2, VES_DEC)
#undef VES_DEC
    }
  }
}

// up1: transposed conv 1 on tiles of v1 vesicles with interleaved rows
// (M = v1 * L/4 = 128), both output parities in one MMA of N = 2*Nd (merged
// image) or two MMAs on the same lanes.  KCD compile-time K chunk count (0:
// from the geometry); NG warp groups (TMEM columns [128*wg, 128*wg + 2*Nd)
// each).  Items are (group, tile) pairs, a.per_grp tiles per group.
// The two warps on a lane quarter take one output parity each.  Its MMAs are
// all math-bound (N = 2*Nd), so the groups issue whole batches in turn: 304 ->
// 262 us (advection), 194 -> 175 us (near field) at 512 vesicles; in down and
// up2, whose batches wait for shared memory, taking turns cost time.
template <int KCD, int NG>
__global__ void __launch_bounds__(NG * kGroupThreads, 1) up1_kernel(KArgs a) {
  extern __shared__ __align__(128) unsigned char sm[];
  __shared__ uint64_t bar[NG], mbar[NG];  // per warp group: MMA completion, intermediate arrival
  __shared__ uint32_t tbase;
  __shared__ int fail[NG], turn;
  const Geo& g = a.g;
  const int kcd = KCD ? KCD : g.kcd;
  const int L = g.L, L2 = L / 2, L4 = L / 4, V1 = g.v1;
  const int ntiles = a.per_grp;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wg = tid / kGroupThreads, gt = tid % kGroupThreads;
  const int qd = warp & 3, r = gt >> 7;  // TMEM lane quarter; the output parity of this warp's epilogue
  const Range rg = my_items(a.items);
  if (rg.lo >= rg.hi) return;
  const uint32_t ncols = 512;
  if (tid == 0) {
    for (int k = 0; k < NG; ++k) {
      tc_mbar_init(&bar[k], 1);
      tc_mbar_init(&mbar[k], 1);
      fail[k] = 0;
    }
    turn = 0;
    tc_mbar_fence_init();
  }
  if (warp == 0) tc_tmem_alloc(&tbase, ncols);
  zero16(sm + g.u1bs, NG * g.u1grp + 128 * 16);  // halos and K padding stay zero
  tc_fence_async_smem();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const int wgu = __shfl_sync(0xffffffffu, wg, 0);  // uniform across the warp
  const bool issuer = __shfl_sync(0xffffffffu, gt >> 5, 0) == 0 && tc_elect();
  const uint32_t dt = __shfl_sync(0xffffffffu, tbase, 0) + (NG == 2 ? 256 : 128) * wgu;
  const uint32_t sbase = tc_smem_u32(sm);
  const float* cst = reinterpret_cast<const float*>(sm + g.u1cst);
  const int PB = (L4 + 4) * V1;  // rows per K chunk: 2*v1 zero rows, the tile's L4*v1 rows, 2*v1 zero rows
  const int Nd = kcd * 8;
  const uint32_t chunk = (uint32_t)(L4 * V1 * 16);  // bytes of one K chunk of a tile
  uint4* bs = reinterpret_cast<uint4*>(sm + g.u1bs + wg * g.u1grp);
  const uint32_t bTap = (uint32_t)((g.u1merge ? 2 * Nd : g.d) * kcd * 16) >> 4;
  const uint32_t lboB1 = (uint32_t)((g.u1merge ? 2 * Nd : g.d) * 16);
  const uint32_t w1 = g.u1merge ? (uint32_t)(g.u1w + Nd * 16) : (uint32_t)(g.u1w + 5 * kcd * g.d * 16);
  // this thread's accumulator row: position q of the tile's vesicle j
  const int row = 32 * qd + lane, q = row / V1, j = row % V1;
  unsigned phase = 0, mphase = 0;
  bool mpend = false;  // a bulk copy into bs is in flight
  // intermediate of a tile [kcd][L/4 * v1][16B] -> bs rows 2*v1 .. (L/4 + 2)*v1 - 1 of each chunk
  auto fetch_mid = [&](int grp, long long t) {
    if (gt == 0) {
      const unsigned char* src = a.mid + ((size_t)t * a.G + grp) * (size_t)V1 * g.mid_bytes;
      tc_expect_tx(&mbar[wg], chunk * (uint32_t)kcd);
      for (int kc = 0; kc < kcd; ++kc) tc_bulk_g2s(bs + kc * PB + 2 * V1, src + (size_t)kc * chunk, chunk, &mbar[wg]);
    }
    mpend = true;
  };
  bool failed = false, stuck = false;
  for (long long lo = rg.lo; lo < rg.hi && !failed;) {
    const Seg sg = next_seg(lo, rg.hi, ntiles);
    __syncthreads();
    copy16(sm, a.img + (size_t)sg.grp * g.u1size, g.u1size);
    tc_fence_async_smem();
    __syncthreads();
    const long long t0 = (long long)sg.grp * ntiles;  // first item of the group
    if (sg.lo + wg < sg.hi) fetch_mid(sg.grp, sg.lo + wg - t0);
    for (long long it = sg.lo + wg; it < sg.hi; it += NG) {
      const long long t = it - t0;
      if (!group_wait_one(&mbar[wg], mphase, a.st, 26, wg, gt, &fail[wg])) {
        failed = true;
        break;
      }
      mphase ^= 1;
      mpend = false;
      tc_fence_after_sync();
      if (issuer) {
        batch_begin(&turn);
        deconv_issue<KCD>(dt, sbase, g.u1bs + wgu * g.u1grp, PB * 16, Nd, kcd, g.u1merge != 0, g.u1w, w1, bTap, lboB1,
                          (uint32_t)V1);
        tc_commit(&bar[wgu]);
        batch_end(&turn);
      }
      if (!group_wait_one(&bar[wg], phase, a.st, 23, wg, gt, &fail[wg])) {
        failed = stuck = true;
        break;
      }
      phase ^= 1;
      tc_fence_after_sync();
      // bs is free once the MMAs have completed: this group's next item
      if (it + NG < sg.hi) fetch_mid(sg.grp, t + NG);
      // output positions 2q + r of vesicle t*v1 + j -> the record of its up2 tile
      const long long v = t * V1 + j;
      const bool own = v < a.nv;
      const int VU = g.vu;
      const long long vs = own ? v : 0;
      uint4* dst = reinterpret_cast<uint4*>(a.mid2 + ((size_t)(vs / VU) * a.G + sg.grp) * (size_t)VU * g.mid2_bytes) +
                   (vs % VU);
#pragma unroll
      for (int k0 = 0; k0 < (KCD ? KCD : 16); k0 += 4) {
        if (k0 >= kcd) break;
        float vv[32];
        tc_ld32(dt + ((uint32_t)(32 * qd) << 16) + r * Nd + 8 * k0, vv);
        if (own) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (k0 + k < kcd)
              dst[((size_t)(k0 + k) * L2 + 2 * q + r) * VU] = act8(vv + 8 * k, cst, k0 + k, g.d, 0, 128, 256);
        }
      }
      tc_fence_before_sync();
      group_sync(wg);  // every TMEM read done before the next item's MMAs
    }
    lo = sg.hi;
    failed = __syncthreads_or(failed ? 1 : 0) != 0;  // every thread takes part
  }
  if (stuck) tc_mbar_wait(&bar[wg], phase, nullptr, 0);
  if (mpend) tc_mbar_wait(&mbar[wg], mphase, nullptr, 0);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tc_tmem_dealloc(tbase, ncols);
}

// up2: transposed conv 2, mix, residual and pass-through, on tiles of VU
// vesicles with interleaved rows (row q*VU + j holds position q of the tile's
// vesicle j).  At L = 128 a tile of two vesicles fills the 128 rows of a
// transposed-conv MMA (one vesicle alone ran M = 64 MMAs at half the math
// rate) and its mix is two MMAs of 128 rows; at L = 256 one vesicle is such a
// tile.
//
// NG warp groups, TMEM columns [cstride*wg, + cstride) each.  The two warps on
// a lane quarter take half of the channel chunks and one of the two mix
// accumulators each.  The residual and the bias go into the mix accumulators
// while the transposed conv runs, straight from global memory (prefetched into
// L2 one item ahead), so the block input needs no shared memory.  The two
// halves of the mix are issued by two threads (one was slower).
template <int KCD, int NG, int VU>
__global__ void __launch_bounds__(NG * kGroupThreads, 1) up2_kernel(KArgs a) {
  extern __shared__ __align__(128) unsigned char sm[];
  __shared__ uint64_t bar[NG], mbar[NG], xbar[NG];  // per warp group: transposed conv, intermediate, mix
  __shared__ uint32_t tbase;
  __shared__ int fail[NG];
  const Geo& g = a.g;
  const int kcd = KCD ? KCD : g.kcd;
  const int L = g.L, L2 = L / 2;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wg = tid / kGroupThreads, gt = tid % kGroupThreads;
  const int qd = warp & 3, hw = gt >> 7;  // TMEM lane quarter; which of the two warps on it
  const int nhalf = VU * L / 128;         // mix accumulators of 128 rows: 2, or 1 (L = 128, VU = 1)
  const Range rg = my_items(a.items);
  if (rg.lo >= rg.hi) return;
  const uint32_t ncols = 512;
  if (tid == 0) {
    for (int k = 0; k < NG; ++k) {
      tc_mbar_init(&bar[k], 1);
      tc_mbar_init(&mbar[k], 1);
      tc_mbar_init(&xbar[k], nhalf);
      fail[k] = 0;
    }
    tc_mbar_fence_init();
  }
  if (warp == 0) tc_tmem_alloc(&tbase, ncols);
  zero16(sm + g.u2cs, NG * g.u2grp + 128 * 16);  // halos and K padding stay zero
  tc_fence_async_smem();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const int Nd = kcd * 8, Nm = rup(g.cmix, 16);
  const int mcol = 2 * Nd;  // mix accumulators: 32 columns each, after the transposed conv's
  // issue from uniform values with tiles of two vesicles only: at L = 256 the
  // faster issue of three groups slowed the kernel (946 -> 1104 us at 512 vesicles)
  constexpr bool kUniform = VU == 2;
  const int wgu = kUniform ? __shfl_sync(0xffffffffu, wg, 0) : wg;
  const int wiu = kUniform ? __shfl_sync(0xffffffffu, gt >> 5, 0) : 0;
  const bool leader = kUniform ? tc_elect() : (gt & 127) == 0;
  const uint32_t dt = (kUniform ? __shfl_sync(0xffffffffu, tbase, 0) : tbase) + (uint32_t)((2 * Nd + 32 * nhalf) * wgu);
  const uint32_t lanes = (uint32_t)(32 * qd) << 16;
  const uint32_t sbase = tc_smem_u32(sm);
  const int goff = wgu * g.u2grp;
  const float* cst = reinterpret_cast<const float*>(sm + g.u2cst);
  const int PC = (L2 + 4) * VU, PD = (L + 2) * VU;
  const int cout = g.cmix + g.npass;
  uint4* cs = reinterpret_cast<uint4*>(sm + g.u2cs + goff);
  uint4* ds = reinterpret_cast<uint4*>(sm + g.u2ds + goff);
  const bool need_x = g.residual || g.npass > 0;
  const uint32_t bTap = (uint32_t)((g.u2merge ? 2 * Nd : g.d) * kcd * 16) >> 4;
  const uint32_t lboB = (uint32_t)((g.u2merge ? 2 * Nd : g.d) * 16);
  const uint32_t w1 = g.u2merge ? (uint32_t)(g.u2w + Nd * 16) : (uint32_t)(g.u2w + 5 * kcd * g.d * 16);
  // this thread's accumulator row: in the transposed conv input position q of
  // the tile's vesicle j, in mix half hw output position pm of the same vesicle
  const int row = 32 * qd + lane, q = row / VU, j = row % VU;
  const int pm = (128 * hw + row) / VU;
  const int ntl = a.per_grp;
  unsigned phase = 0, mphase = 0, xphase = 0;
  bool mpend = false, dpend = false, xpend = false;  // bulk copy into cs, transposed conv, mix in flight
  // up1 output [kcd][L/2 * VU][16B] of tile t -> cs rows 2*VU .. (L/2 + 2)*VU - 1 of each chunk
  auto fetch_mid = [&](int grp, long long t) {
    if (gt == 0) {
      const unsigned char* src = a.mid2 + ((size_t)t * a.G + grp) * (size_t)VU * g.mid2_bytes;
      tc_expect_tx(&mbar[wg], (uint32_t)(VU * g.mid2_bytes));
      for (int kc = 0; kc < kcd; ++kc)
        tc_bulk_g2s(cs + kc * PC + 2 * VU, src + (size_t)kc * L2 * VU * 16, (uint32_t)(L2 * VU * 16), &mbar[wg]);
    }
    mpend = true;
  };
  // block input x[v][grp*cin + c][pos] of tile t -> L2
  auto fetch_x = [&](int grp, long long t) {
    const long long v = t * VU + (gt - 32);
    if (gt >= 32 && gt < 32 + VU && v < a.nv)
      tc_prefetch_l2(a.x + (v * a.G + grp) * (long long)g.cin * L, (uint32_t)(g.cin * L * 4));
  };
  bool failed = false;
  for (long long lo = rg.lo; lo < rg.hi && !failed;) {
    const Seg sg = next_seg(lo, rg.hi, ntl);
    __syncthreads();
    copy16(sm, a.img + (size_t)sg.grp * g.u2size, g.u2size);
    tc_fence_async_smem();
    __syncthreads();
    const long long t0 = (long long)sg.grp * ntl;  // first item of the group
    if (sg.lo + wg < sg.hi) {
      fetch_mid(sg.grp, sg.lo + wg - t0);
      if (need_x) fetch_x(sg.grp, sg.lo + wg - t0);
    }
    for (long long it = sg.lo + wg; it < sg.hi; it += NG) {
      const long long v = (it - t0) * VU + j;
      const bool on = hw < nhalf && v < a.nv;
      const long long vs = v < a.nv ? v : 0;
      const float* __restrict__ xp = a.x + (vs * a.G + sg.grp) * (long long)g.cin * L + pm;
      float* __restrict__ op = a.out + (vs * a.G + sg.grp) * (long long)cout * L + pm;
      if (!group_wait_one(&mbar[wg], mphase, a.st, 26, wg, gt, &fail[wg])) {
        failed = true;
        break;
      }
      mphase ^= 1;
      mpend = false;
      tc_fence_after_sync();  // every TMEM read of the previous item is done
      if (kUniform ? wiu == 0 && leader : gt == 0) {
        deconv_issue<KCD>(dt, sbase, g.u2cs + goff, PC * 16, Nd, kcd, g.u2merge != 0, g.u2w, w1, bTap, lboB, VU);
        tc_commit(&bar[wgu]);
      }
      dpend = true;
      if (need_x && it + NG < sg.hi) fetch_x(sg.grp, it + NG - t0);
      if (hw < nhalf) {
        // mix accumulator hw preset to residual + bias while the transposed conv runs
        float r0[32];
#pragma unroll
        for (int o = 0; o < 32; ++o) r0[o] = (o < g.cmix && g.residual && on) ? __ldg(xp + o * L) : 0.f;
#pragma unroll
        for (int o = 0; o < 32; ++o) r0[o] = r0[o] + (o < g.cmix ? cst[768 + o] : 0.f);
        tc_st32(dt + lanes + mcol + 32 * hw, r0);
        // pass-through channels
        if (on)
          for (int c = 0; c < g.npass; ++c) op[(g.cmix + c) * L] = __ldg(xp + (g.cin - g.npass + c) * L);
        tc_wait_st();
      }
      if (!group_wait_one(&bar[wg], phase, a.st, 24, wg, gt, &fail[wg])) {
        failed = true;
        break;
      }
      phase ^= 1;
      dpend = false;
      tc_fence_after_sync();
      // cs is free once the transposed conv has completed: this group's next item
      if (it + NG < sg.hi) fetch_mid(sg.grp, it + NG - t0);
      if (32 * qd < L2 * VU) {  // uniform per warp
        const bool own = row < L2 * VU;
        const int k1 = hw ? kcd : kcd / 2;
        if (VU == 2) {
          // both parities of two chunks at a time: one read of the constants serves both
#pragma unroll
          for (int kk = 0; kk < (KCD ? KCD / 2 : 8); kk += 2) {
            const int k0 = hw * (kcd / 2) + kk;
            if (k0 >= k1) break;
            float vv[32];
            tc_ld16x2(dt + lanes + 8 * k0, dt + lanes + Nd + 8 * k0, vv);
            if (own) {
#pragma unroll
              for (int k = 0; k < 2; ++k)
                if ((KCD == 0 || kk + k < KCD / 2) && k0 + k < k1) {
                  const uint4 e0 = act8(vv + 8 * k, cst, k0 + k, g.d, 384, 512, 640);
                  const uint4 e1 = act8(vv + 16 + 8 * k, cst, k0 + k, g.d, 384, 512, 640);
                  uint4* o = ds + (size_t)(k0 + k) * PD + (2 * q + 1) * VU + j;
                  o[0] = e0;
                  o[VU] = e1;
                }
            }
          }
        } else {
          // one parity at a time (80 registers with three groups)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
#pragma unroll
            for (int kk = 0; kk < (KCD ? KCD / 2 : 8); kk += 4) {
              const int k0 = hw * (kcd / 2) + kk;
              if (k0 >= k1) break;
              float vv[32];
              tc_ld32(dt + lanes + r * Nd + 8 * k0, vv);
              if (own) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                  if ((KCD == 0 || kk + k < KCD / 2) && k0 + k < k1)
                    ds[(size_t)(k0 + k) * PD + (2 * q + r + 1) * VU + j] = act8(vv + 8 * k, cst, k0 + k, g.d, 384, 512, 640);
              }
            }
          }
        }
      }
      group_sync_for_mma(wg);
      // mix: D[p][o] = sum_t d[p + t - 1] M_t onto residual + bias, 128 rows per issuing thread
      if (leader && hw < nhalf && (!kUniform || (wiu & 3) == 0)) {
        const uint32_t idesc = tc_idesc_bf16(128, Nm);
        const uint32_t lboA = PD * 16, lboM = g.cmix * 16;
        const uint64_t a0 = tc_desc(sbase + g.u2ds + goff, lboA, 128), b0 = tc_desc(sbase + g.u2wm, lboM, 128);
        const uint32_t hh = kUniform ? (uint32_t)wiu >> 2 : (uint32_t)hw;
#define VES_MIX(NK) issue_mix<NK>(dt + mcol + 32 * hh, a0 + 128 * hh, b0, (kcd * lboM) >> 4, (2 * lboA) >> 4, (2 * lboM) >> 4, idesc, VU)
        VES_TC_NK_SWITCH(kcd / 2, VES_MIX)
#undef VES_MIX
        tc_commit(&xbar[wgu]);
      }
      xpend = true;
      if (!group_wait_one(&xbar[wg], xphase, a.st, 25, wg, gt, &fail[wg])) {
        failed = true;
        break;
      }
      xphase ^= 1;
      xpend = false;
      tc_fence_after_sync();
      if (hw < nhalf) {
        float vv[32];
        tc_ld32(dt + lanes + mcol + 32 * hw, vv);
        if (on) {
#pragma unroll
          for (int o = 0; o < 32; ++o)
            if (o < g.cmix) op[o * L] = vv[o];
        }
      }
      tc_fence_before_sync();
      group_sync(wg);
    }
    lo = sg.hi;
    failed = __syncthreads_or(failed ? 1 : 0) != 0;  // every thread takes part
  }
  // bounded drains: this group's MMAs and bulk copies still in flight after a failure
  if (dpend) tc_mbar_wait(&bar[wg], phase, nullptr, 0);
  if (xpend) tc_mbar_wait(&xbar[wg], xphase, nullptr, 0);
  if (mpend) tc_mbar_wait(&mbar[wg], mphase, nullptr, 0);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tc_tmem_dealloc(tbase, ncols);
}

}  // namespace tcnet


// ---------------------------------------------------------------------------
// host side
#include "ves_nets_tc.h"

namespace {

uint16_t bf16_rn(float f) {
  uint32_t u;
  memcpy(&u, &f, 4);
  if ((u & 0x7f800000u) == 0x7f800000u) return (uint16_t)(u >> 16);  // inf / nan
  const uint32_t lsb = (u >> 16) & 1u;
  u += 0x7fffu + lsb;
  return (uint16_t)(u >> 16);
}

void put_row(unsigned char* img, size_t off, const float* vals8) {
  uint16_t* p = reinterpret_cast<uint16_t*>(img + off);
  for (int e = 0; e < 8; ++e) p[e] = bf16_rn(vals8[e]);
}

}  // namespace

int tcnet_pack(const ves_net_block& b, int G, int L, const float* const* p, std::vector<unsigned char>& down,
               std::vector<unsigned char>& up1, std::vector<unsigned char>& up2, TcBlock& out) {
  using namespace tcnet;
  const Geo g = make_geo(b, L);
  static_assert(sizeof(Geo) <= sizeof(out.geo), "geometry record too large");
  out.geo_bytes = sizeof(Geo);
  memcpy(out.geo, &g, sizeof(Geo));
  out.dsize = g.dsize;
  out.u1size = g.u1size;
  out.u2size = g.u2size;
  out.mid_bytes = g.mid_stride;
  // TMEM per warp group with two groups (256 columns each): N1 + N2 (down),
  // 2 * Nd (up1) and 2 * Nd + the mix halves (up2); the mix epilogue reads 32
  // columns; each lane quarter holds 32 whole positions; every kernel fits
  // two warp groups in shared memory
  if (g.n1 > 128 || g.d > 128 || g.cmix > 32 || 2 * g.kcd * 8 + (L / 128) * rup(g.cmix, 16) > 256 ||
      g.dxs + 2 * g.dgrp + kTail > kMaxSmem || g.u1size + 2 * g.u1grp + kTail > kMaxSmem ||
      g.u2size + 2 * g.u2grp + kTail > kMaxSmem || L > 256 || (L / 4) % 32 != 0)
    return VES_ERR_ARG;
  const int c1 = b.c1, c2 = b.c2, d = g.d, cin = b.cin, cmix = b.cmix;
  down.assign((size_t)g.dsize * G, 0);
  up1.assign((size_t)g.u1size * G, 0);
  up2.assign((size_t)g.u2size * G, 0);
  auto bn = [&](int idx, int ch, float* s, float* t) {
    const float* w = p[14 + 4 * idx];
    const float* bb = p[15 + 4 * idx];
    const float* mean = p[16 + 4 * idx];
    const float* var = p[17 + 4 * idx];
    const double inv = 1.0 / std::sqrt((double)var[ch] + 1e-5);
    *s = (float)((double)w[ch] * inv);
    *t = (float)((double)bb[ch] - (double)mean[ch] * (double)w[ch] * inv);
  };
  for (int grp = 0; grp < G; ++grp) {
    unsigned char* D = down.data() + (size_t)grp * g.dsize;
    unsigned char* U1 = up1.data() + (size_t)grp * g.u1size;
    unsigned char* U2 = up2.data() + (size_t)grp * g.u2size;
    float v8[8];
    // conv pair 1
    for (int oi = 0; oi < kOffsets; ++oi) {
      const int s = shift_of(oi);
      for (int kc = 0; kc < g.kcin; ++kc)
        for (int o = 0; o < g.n1; ++o) {
          for (int e = 0; e < 8; ++e) {
            const int c = kc * 8 + e;
            float w = 0.f;
            if (c < cin) {
              if (o < c1) {
                const int t = s + 3;
                if (t >= 0 && t < 7) w = p[0][((size_t)(grp * c1 + o) * cin + c) * 7 + t];
              } else if ((s & 1) == 0) {
                const int t = (s + 6) / 2;
                w = p[2][((size_t)(grp * c1 + o - c1) * cin + c) * 7 + t];
              }
            }
            v8[e] = w;
          }
          put_row(D, g.dw1 + ((size_t)(oi * g.kcin + kc) * g.n1 + o) * 16, v8);
        }
      for (int kc = 0; kc < g.kc1; ++kc)
        for (int o = 0; o < d; ++o) {
          for (int e = 0; e < 8; ++e) {
            const int c = kc * 8 + e;
            float w = 0.f;
            if (c < g.n1) {
              if (o < c2) {
                const int t = s + 3;
                if (t >= 0 && t < 7) w = p[4][((size_t)(grp * c2 + o) * g.n1 + c) * 7 + t];
              } else if ((s & 1) == 0) {
                const int t = (s + 6) / 2;
                w = p[6][((size_t)(grp * c2 + o - c2) * g.n1 + c) * 7 + t];
              }
            }
            v8[e] = w;
          }
          put_row(D, g.dw2 + ((size_t)(oi * g.kc1 + kc) * d + o) * 16, v8);
        }
    }
    float* dc = reinterpret_cast<float*>(D + g.dcst);
    for (int o = 0; o < g.n1; ++o) {
      dc[o] = o < c1 ? p[1][grp * c1 + o] : p[3][grp * c1 + o - c1];
      bn(0, grp * g.n1 + o, &dc[128 + o], &dc[256 + o]);
    }
    for (int o = 0; o < d; ++o) {
      dc[384 + o] = o < c2 ? p[5][grp * c2 + o] : p[7][grp * c2 + o - c2];
      bn(1, grp * d + o, &dc[512 + o], &dc[640 + o]);
    }
    // transposed convs: A[o][c] = W[grp*d + c][o][r + 2u]
    for (int layer = 0; layer < 2; ++layer) {
      const float* W = p[8 + 2 * layer];
      for (int r = 0; r < 2; ++r)
        for (int u = 0; u < 5; ++u)
          for (int kc = 0; kc < g.kcd; ++kc)
            for (int o = 0; o < d; ++o) {
              for (int e = 0; e < 8; ++e) {
                const int c = kc * 8 + e;
                v8[e] = c < d ? W[((size_t)(grp * d + c) * d + o) * 10 + r + 2 * u] : 0.f;
              }
              if (layer == 0)
                put_row(U1, g.u1merge ? dec_w_off_merged(g, g.u1w, r, u, kc, o) : dec_w_off(g, g.u1w, r, u, kc, o),
                        v8);
              else if (g.u2merge)
                put_row(U2, dec_w_off_merged(g, g.u2w, r, u, kc, o), v8);
              else
                put_row(U2, dec_w_off(g, g.u2w, r, u, kc, o), v8);
            }
    }
    for (int t = 0; t < 3; ++t)
      for (int kc = 0; kc < g.kcd; ++kc)
        for (int o = 0; o < cmix; ++o) {
          for (int e = 0; e < 8; ++e) {
            const int c = kc * 8 + e;
            v8[e] = c < d ? p[12][((size_t)(grp * cmix + o) * d + c) * 3 + t] : 0.f;
          }
          put_row(U2, g.u2wm + ((size_t)(t * g.kcd + kc) * cmix + o) * 16, v8);
        }
    float* uc = reinterpret_cast<float*>(U1 + g.u1cst);
    for (int o = 0; o < d; ++o) {
      uc[o] = p[9][grp * d + o];
      bn(2, grp * d + o, &uc[128 + o], &uc[256 + o]);
      uc[384 + o] = p[11][grp * d + o];
      bn(3, grp * d + o, &uc[512 + o], &uc[640 + o]);
    }
    for (int o = 0; o < cmix; ++o) uc[768 + o] = p[13][grp * cmix + o];
    memcpy(U2 + g.u2cst, U1 + g.u1cst, 7 * 128 * 4);  // both up kernels carry the full constants block
  }
  return VES_OK;
}

namespace {

// compiled chunk-count variants; others run the generic kernels
void (*pick_down(int kc1, int kcd, int ng, int vd))(tcnet::KArgs) {
  using namespace tcnet;
#define VES_DK(A, B, V) return ng == 3 ? down_kernel<A, B, 3, V> : down_kernel<A, B, 2, V>
  if (vd == 1) {
    if (kc1 == 4 && kcd == 6) VES_DK(4, 6, 1);
    VES_DK(0, 0, 1);
  }
  if (kc1 == 6 && kcd == 6) VES_DK(6, 6, 2);
  if (kc1 == 6 && kcd == 8) VES_DK(6, 8, 2);
  if (kc1 == 8 && kcd == 8) VES_DK(8, 8, 2);
  VES_DK(0, 0, 2);
#undef VES_DK
}

void (*pick_up1(int kcd, int ng))(tcnet::KArgs) {
  using namespace tcnet;
  if (kcd == 6) return ng == 3 ? up1_kernel<6, 3> : up1_kernel<6, 2>;
  if (kcd == 8) return ng == 3 ? up1_kernel<8, 3> : up1_kernel<8, 2>;
  return ng == 3 ? up1_kernel<0, 3> : up1_kernel<0, 2>;
}

void (*pick_up2(int kcd, int ng, int vu))(tcnet::KArgs) {
  using namespace tcnet;
  if (vu == 2) return kcd == 6 ? (ng == 3 ? up2_kernel<6, 3, 2> : up2_kernel<6, 2, 2>)
                               : (kcd == 8 ? up2_kernel<8, 2, 2> : up2_kernel<0, 2, 2>);
  if (kcd == 6 && ng > 1) return ng == 3 ? up2_kernel<6, 3, 1> : up2_kernel<6, 2, 1>;
  return ng == 1 ? up2_kernel<0, 1, 1> : up2_kernel<0, 2, 1>;
}

bool autotune_log() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("VES_TC_AUTOTUNE_LOG");
    v = (e && atoi(e)) ? 1 : 0;
  }
  return v != 0;
}

}  // namespace

int tcnet_run_block(const TcBlock& tb, int G, int nv, const unsigned char* d_down, const unsigned char* d_up1,
                    const unsigned char* d_up2, const float* x, float* out, unsigned char* mid, VesDeviceStatus* st,
                    cudaStream_t s, bool autotune) {
  using namespace tcnet;
  // the block input and the intermediates are fetched by 16-byte bulk copies
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(mid)) & 15u) {
    ves_record_error(VES_ERR_ARG, "net_forward: input and workspace must be 16-byte aligned");
    return VES_ERR_ARG;
  }
  KArgs a;
  memcpy(&a.g, tb.geo, sizeof(Geo));
  const Geo& g = a.g;
  a.G = G;
  a.nv = nv;
  a.items = (long long)G * nv;
  a.x = x;
  a.out = out;
  a.per_grp = nv;
  const int ntiles = (nv + g.v1 - 1) / g.v1;
  a.mid = mid;
  a.mid2 = mid + (size_t)ntiles * G * g.v1 * g.mid_bytes;
  a.st = st;
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int kc1 = g.kc1, kcd = g.kcd, Nd = kcd * 8;
  // warp groups per CTA that fit: TMEM (512 columns) and shared memory
  const int down3 = g.dxs + 3 * g.dgrp + kTail, up1_3 = g.u1size + 3 * g.u1grp + kTail, up2_3 = g.u2size + 3 * g.u2grp + kTail;
  const int ucols = 2 * Nd + 32 * (g.vu * g.L / 128);  // TMEM columns per up2 group
  const bool dn3 = (kc1 + kcd) * 8 <= 128 && down3 <= kMaxSmem;
  const bool u13 = 2 * Nd <= 128 && up1_3 <= kMaxSmem;
  const bool u22 = 2 * ucols <= 512, u23 = kcd == 6 && 3 * ucols <= 512 && up2_3 <= kMaxSmem;
  const int grid = (int)std::min<long long>(a.items, (long long)nsm);
  // one CTA per SM (it allocates all 512 TMEM columns): at least 117 KB of
  // shared memory per CTA keeps a second one off the SM
  auto launch = [&](int which, int ng) -> int {
    KArgs b = a;
    void (*fn)(KArgs);
    int smem;
    int nblk = grid;
    if (which == 0) {
      fn = pick_down(kc1, kcd, ng, g.vd);
      smem = std::max(g.dxs + ng * g.dgrp + kTail, kMinSmem);
      b.img = d_down;
      b.per_grp = (nv + g.vd - 1) / g.vd;  // items: (group, tile of vd vesicles)
      b.items = (long long)G * b.per_grp;
      nblk = (int)std::min<long long>(b.items, (long long)nsm);
    } else if (which == 1) {
      fn = pick_up1(kcd, ng);
      smem = std::max(g.u1size + ng * g.u1grp + kTail, kMinSmem);
      b.img = d_up1;
      b.per_grp = ntiles;  // items: (group, tile)
      b.items = (long long)G * ntiles;
      nblk = (int)std::min<long long>(b.items, (long long)nsm);
    } else {
      fn = pick_up2(kcd, ng, g.vu);
      smem = std::max(g.u2size + ng * g.u2grp + kTail, kMinSmem);
      b.img = d_up2;
      b.per_grp = (nv + g.vu - 1) / g.vu;  // items: (group, tile of vu vesicles)
      b.items = (long long)G * b.per_grp;
      nblk = (int)std::min<long long>(b.items, (long long)nsm);
    }
    int rc = ves_cuda_status(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                             "tc smem attribute");
    if (rc) return rc;
    ves_count_launch();
    fn<<<nblk, ng * kGroupThreads, smem, s>>>(b);
    return ves_launch_check("tc net block");
  };
  // the fixed rule: the most warp groups that fit
  TcPlan plan{nv, dn3 ? 3 : 2, u13 ? 3 : 2, u23 ? 3 : (u22 ? 2 : 1)};
  const TcPlan* found = nullptr;
  for (const TcPlan& p : tb.plans)
    if (p.nv == nv) found = &p;
  if (found) {
    plan = *found;
  } else if (autotune) {
    cudaEvent_t e0, e1;
    int rc = ves_cuda_status(cudaEventCreate(&e0), "tune event");
    if (!rc) rc = ves_cuda_status(cudaEventCreate(&e1), "tune event");
    if (rc) return rc;
    auto timed = [&](int which, int ng, float& ms) -> int {
      ms = 1e30f;
      for (int rep = 0; rep < 2; ++rep) {
        int r = ves_cuda_status(cudaEventRecord(e0, s), "tune record");
        if (!r) r = launch(which, ng);
        if (!r) r = ves_cuda_status(cudaEventRecord(e1, s), "tune record");
        if (!r) r = ves_cuda_status(cudaEventSynchronize(e1), "tune sync");
        float t = 0.f;
        if (!r) r = ves_cuda_status(cudaEventElapsedTime(&t, e0, e1), "tune elapsed");
        if (r) return r;
        ms = std::min(ms, t);
      }
      return VES_OK;
    };
    float best = 1e30f, t = 0.f;
    // each kernel in the order the block runs them, so that the next one reads a valid input
    for (int ng = 2; ng <= 3 && !rc; ++ng) {
      if (ng == 3 && !dn3) continue;
      if ((rc = timed(0, ng, t))) break;
      if (t < best) best = t, plan.ng_down = ng;
    }
    if (!rc) rc = launch(0, plan.ng_down);
    best = 1e30f;
    for (int ng = 2; ng <= 3 && !rc; ++ng) {
      if (ng == 3 && !u13) continue;
      if ((rc = timed(1, ng, t))) break;
      if (t < best) best = t, plan.ng_up1 = ng;
    }
    if (!rc) rc = launch(1, plan.ng_up1);
    best = 1e30f;
    for (int ng = u22 ? 2 : 1; ng <= 3 && !rc; ++ng) {
      if ((ng == 2 && !u22) || (ng == 3 && !u23)) continue;
      if ((rc = timed(2, ng, t))) break;
      if (t < best) best = t, plan.ng_up2 = ng;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    tb.plans.push_back(plan);
    if (autotune_log())
      fprintf(stderr, "tcnet autotune: L=%d kc1=%d kcd=%d nv=%d -> down %d groups, up1 %d groups, up2 %d groups\n", g.L,
              kc1, kcd, nv, plan.ng_down, plan.ng_up1, plan.ng_up2);
  }
  int rc = launch(0, plan.ng_down);
  if (!rc) rc = launch(1, plan.ng_up1);
  if (!rc) rc = launch(2, plan.ng_up2);
  return rc;
}
