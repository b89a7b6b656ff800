// ocn_slice.cu -- the FP64 contractions of the BSE action on the FP8 tensor cores.
//
//   phi(k,x,t)    = sum_n u(n,k,x) q(n,k,t)              (band -> x)
//   part(n,k,t)   = - sum_x conj(u(n,k,x)) phi'(k,x,t)   (x -> band)
//
// GB300 issues FP64 at 2 fused multiply-adds per clock and SM, so on the FP64
// pipe these two sums cost 4.3 and 5.9 ms on the 8^3 k / 100-band / 12^3 x case
// while their operands could be read in 0.2 ms.  Here every operand row (a row of
// u over the summed index, a column of q or phi') is written as a binary fixed
// point number of 60 bits against the largest exponent of the row, cut into
// S = 12 signed base-32 digits (|d| <= 16, exact in E4M3), and
//   sum a b = 2^(ea + eb - 118) sum_(i,j) 32^(22-i-j) sum_K d_i(a) d_j(b)
// is formed on the tensor cores.  |d_i d_j| <= 256, so the FP32 accumulator of a
// group i + j is an exact integer while K * pairs * 256 <= 2^24 (x -> band: kept by
// the choice of the K splits; band -> x, which has none: by the largest number of
// bands, asserted below); the groups i + j <= 12 are added in 64-bit integers
// and rounded to binary64 once (per K split).
//
// Accuracy.  What is left out are digits below 2^-60 of a row's largest element and
// pairs with i + j > 12.  For rows whose elements are of one size that is a tenth of
// the rounding error of an FP64 sum; where a row is small at the K at which the column
// is large it would not be.  The epilogue checks every sum (see check_part) and forms
// those that the digits do not hold as well in binary64.  An action is therefore as
// accurate as an FP64 one element by element, not only in the norm.  (With the groups
// i + j <= 11 the check left many sums over preconditioned GMRES residuals open, which
// are peaked over the bands: the 64 k / 32 bands gradient took 220 ms, now 130.)
//
// The sums of a K split are exact; splits are rounded and added one after another, and
// chunks and splits follow the context's largest block (nvec), so results do not depend
// on the vectors that share a launch, but may differ in the last bit between contexts.
//
// Layout.  The digits of u are stored in the order in which the kernel consumes
// them, as no-swizzle K-major core matrices ([granule of 16 K][row][16 bytes]), so
// every pipeline stage is one contiguous bulk copy:
//   A[spin][k][row tile of 128][K chunk][box][granule][row][16]
// box = slice (band -> x: K runs over re n then im n) or plane * 12 + slice (x ->
// band: re and im planes of u, K over x).  12 bytes per real against 8 for FP64, and
// one byte per complex element of magnitudes for the check.
// The vector side is small and rebuilt per action:
//   B[k][granule][part][slice][column][16]
// In shared memory each granule's digit rows follow 11 empty slices, so the
// operand of slice i of A is the same buffer read from row (11 - i) C: its digit j
// meets output column group i + j, and one MMA of N = 13 C columns per (slice, 32
// K) adds every pair of that slice.  part: re/im columns; both in one MMA (C = 2
// columns each) with up to 8 columns, else one MMA per part (x -> band swaps the
// parts between the planes and negates A for the last of the four).
// The kernel is persistent and warp-specialised like k_lr_tc; CTAs take
// contiguous tile ranges so that the B operand of a k-point is read once.
//
// Measured, 8^3 k / 100 bands / 12^3 x, 1s: band -> x 4.3 ms on the FP64 pipe ->
// 0.345 ms (2.3 GB, 6.7 TB/s), x -> band 5.9 ms -> 0.355 ms (6.4 TB/s): bound by
// the read of A.  2p, 6^3 k / 64 bands / 10^3 x (12 columns): 0.099 and 0.108 ms
// (3.5 and 3.2 TB/s): there the 160-column MMAs (80 cycles) and the epilogue's
// 312 integer columns per row weigh as much as the 0.33 GB read.  Without the group
// i + j = 12 and the check the four took 0.331, 0.355, 0.083 and 0.104 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <new>
#include <string>

#include "ocn_fixed.cuh"
#include "ocn_internal.h"
#include "ocn_tc.cuh"

namespace ocn {

namespace {

constexpr int SL_S = 12;           // digits per value
constexpr int SL_FRAC = 59;        // fixed point: t = v 2^(59 - e), |v| < 2^e
constexpr int SL_ROWS = 128;       // rows per tile (MMA M)
// MMA N: the 13 groups i + j <= 12 of C columns, in steps of 16
__host__ __device__ constexpr int slice_n(int C) { return (13 * C + 15) / 16 * 16; }
// Rows of a granule of B in shared memory: 11 empty and 12 digit slices per part, and empty rows
// to the end of the last part's widest operand (the other part's ends in the next empty slices)
__host__ __device__ constexpr int slice_rows(int C, int P) { return (P - 1) * 23 * C + 11 * C + slice_n(C); }
// Two control warps and four epilogue warps; eight with 8 or 12 columns, half of the
// columns each (band -> x of the 2p case: 113 us with four warps and 255 registers,
// 84 us with eight).
constexpr int slice_threads(int nae) { return nae == 4 ? 192 : 320; }
// (1s case of 512 k / 100 bands, x -> band: 355 us with six stages, 369 us with seven)
constexpr int SL_MAX_STAGES = 6;
constexpr size_t SL_SMEM = 222 * 1024;
constexpr int SL_MAX_K = 2730;      // K per plane and accumulation: 2 * 2730 * 12 * 256 < 2^24
static_assert(OCN_MAX_NB <= SL_MAX_K, "band -> x sums 2 Nb products (re n, im n) in one accumulation");
constexpr unsigned long long SL_BIAS = 0x0842108421084210ull;  // sum of 16 * 32^i, i < 12

struct SliceParams {
  const uint8_t *A, *B;
  const int *eA, *eB;
  int nk, rows, nt, rl, R;   // rows of A per k; row tiles; rows of the last tile and of a k-point (multiples of 8)
  int G, Ge, KC, nch;        // 16-wide K granules (A; B padded to even), granules per chunk, chunks
  int ks, cps;               // K splits, chunks per split
  int ntiles, stages;
  int sb;                    // boxes (slices) per pipeline stage, a divisor of 12
  uint32_t stage_bytes;
  int bshared, koff, spin;   // B one k slice for all k; added to k for A; -1 or the spin whose columns are written
  int na, nvw;               // channels per vector; vectors written
  double2* phi;              // band -> x: [k][row][t]
  double* part;              // x -> band: [split][vector][re|im][npsi]
  size_t part_stride, npsi;
  int nb;
  int negate;                // x -> band: the long-range term subtracts, the multiplet back-projection adds
  int starve;                // test hook: the load warp issues nothing, so the MMA warp's bounded wait runs out
  int* err;
  // the check of the sums and its binary64 fallback
  const uint4* A8;           // magnitudes of u (k_slice_build_mag)
  const uint2* B8;           // and of the columns, [k][t][32 S8 bytes]
  int K, S8;                 // complex products of a sum; steps of 32 of them
  int sample, least;         // steps of the first pass and the least sum that clears
  const double2* u;          // of this spin, element (x, k, n) at x*ux + k*uk + n
  size_t ux, uk;
  const double *pr, *pi, *allow;  // band -> x: psi of the columns
  size_t vstride;
  const double2* f;          // x -> band: [k][x][t], integers with exponents ex[x][t] or binary64
  const int* ex;
};

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// K-major operand without swizzling: 8-row core matrices of 128 bytes (stride
// byte offset 128), consecutive 16-byte K granules lbo bytes apart.
// Low word of the descriptor; addresses stay below 2^18, so adding (bytes >> 4)
// moves the start address.  The high word is the same for every operand.
__device__ __forceinline__ uint32_t plain_desc(uint32_t saddr, uint32_t lbo) {
  return ((saddr >> 4) & 0x3FFFu) | ((lbo >> 4) << 16);
}
constexpr uint32_t PLAIN_DESC_HI = (128 >> 4) | (1u << 14);
__device__ __forceinline__ void umma_fp8(uint32_t dtmem, uint32_t adesc, uint32_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
      "mov.b64 a, {%1, %5};\n\t"
      "mov.b64 b, {%2, %5};\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a, b, %3, p;\n\t}" ::"r"(dtmem),
      "r"(adesc), "r"(bdesc), "r"(idesc), "r"(accumulate), "r"(PLAIN_DESC_HI)
      : "memory");
}
// A (4 or 6) consecutive accumulator columns of this thread's lane
template <int A>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, float* v) {
  static_assert(A == 4 || A == 6, "4 or 6 columns");
  uint32_t r[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
  if constexpr (A == 6) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr + 4));
    v[4] = __uint_as_float(r[0]);
    v[5] = __uint_as_float(r[1]);
  }
}

// NG accumulator groups (most significant first, stride C columns) of A columns as integers.
template <int A, int C, int NG>
__device__ __forceinline__ void add_groups(uint32_t ta, long long (&acc)[A]) {
  float v[NG * A];
#pragma unroll
  for (int g = 0; g < NG; ++g) tmem_ld_cols<A>(ta + g * C, v + g * A);
  tmem_ld_wait();
#pragma unroll
  for (int c = 0; c < A; ++c) acc[c] = 0;
#pragma unroll
  for (int g = 0; g < NG; ++g)
#pragma unroll
    for (int c = 0; c < A; ++c)
      acc[c] += (long long)__float2int_rn(v[g * A + c]) * (long long)(1 << (5 * (NG - 1 - g)));
}

struct SliceTile {
  int k, mt, sp, c0, c1, rt;
};
template <int MODE>
__device__ __forceinline__ SliceTile slice_decode(const SliceParams& p, int t) {
  SliceTile ti;
  const int per_k = p.nt * p.ks;
  ti.k = t / per_k;
  const int r = t - ti.k * per_k;
  ti.mt = r / p.ks;
  ti.sp = r - ti.mt * p.ks;
  ti.c0 = ti.sp * p.cps;
  ti.c1 = min(p.nch, ti.c0 + p.cps);
  ti.rt = ti.mt == p.nt - 1 ? p.rl : SL_ROWS;
  return ti;
}

// x w for a mask weight w, without the FP64 pipe where w = 1
__device__ __forceinline__ double weigh(double x, double w) {
  const long long b = __double_as_longlong(w);
  if (b == 0x3ff0000000000000ll) return x;
  return x * w;
}

// ------------------------------------------------------ graded rows and columns

// The digits of a row and of a column end at 2^-60 of their largest elements.  A sum whose
// terms are all small against the product of the two maxima -- row and column graded
// oppositely -- would be less accurate than in binary64.  The epilogue bounds sum |a||b| of
// every sum from below by 8-bit magnitudes, and the sums that the bound does not clear are
// formed in binary64 from u and the column after the CTA's tiles.
//
// The error of a digit sum of K complex products is sqrt(2) 2^-60.8 (2^eb |a|_2 + 2^ea |b|_2)
// (the two in quadrature; rounding of the elements) and 2^-64.8 sqrt(2 K) 2^(ea + eb) (pairs
// left out) per part.  A sum is cleared when this is at most a quarter of 2^-53 sum |a||b|;
// sums of products in binary64 are off by 0.3 to 0.5 of that (K = 4..1000).  In magnitudes m
// (2^e = 256): (sum m(a) m(b))^2 >= 42 (sum m(a)^2 + sum m(b)^2) + 10100 K.  Ungraded Gaussian
// rows have 18 (K = 1) to 150 (K = 500) times the square root of that, rows graded oppositely
// over two decades about as much.
constexpr float SL_CHECK_M = 42.0f, SL_CHECK_K = 10100.0f;

__device__ __forceinline__ void mma_u8(int (&c)[4], const uint4& a, const uint2& b) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a.x), "r"(a.z), "r"(a.y), "r"(a.w), "r"(b.x), "r"(b.y));
}
// exponent of a row or column whose sums are checked: not of zeros (or subnormal), Inf or NaN
__device__ __forceinline__ bool plain_exp(int e) { return e > -1022 && e != FX_NAN; }
// A warp checks the AH <= 8 columns from h0 on that its threads drain, one column tile of the MMA.
template <int NAE, int AH>
__device__ __forceinline__ unsigned plain_columns(const SliceParams& p, int k, int h0) {
  const int lane = threadIdx.x & 31, t = h0 + min(lane, AH - 1);
  const int e = p.eB[(p.bshared ? 0 : (size_t)k) * NAE + t];
  return __ballot_sync(0xffffffffu, lane < AH && plain_exp(e) && (p.spin < 0 || (t & 1) == p.spin));
}
// this lane's words of its column; columns beyond the last repeat it
template <int NAE, int AH>
__device__ __forceinline__ const uint2* check_column(const SliceParams& p, int k, int h0) {
  const int lane = threadIdx.x & 31;
  return p.B8 + ((p.bshared ? 0 : (size_t)k) * NAE + h0 + min(lane >> 2, AH - 1)) * p.S8 * 4 + (lane & 3);
}

// First pass, by a warp for the 32 rows of group rg: part of K (p.sample steps of 32) against
// the largest error that any row and column of K elements can have, (sum)^2 >= K (2 * 42 *
// 255^2 + 10100).  A partial sum bounds the whole from below; ungraded rows pass about ten
// times over, so the magnitudes are read in part (512 k / 100 bands / 12^3 x: 57 and 17 of
// 113 MB each) while the tile's digits are still on their way.  As a kernel of its own
// after the contraction the check took 18 and 10 us and a launch each.
template <int NAE, int AH>
__device__ __forceinline__ bool check_part(const SliceParams& p, int k, int rg, int h0) {
  const int lane = threadIdx.x & 31, lg = lane >> 2, lq = lane & 3, ngrp = (p.rows + 31) / 32;
  if (rg >= ngrp) return true;
  const uint4* A = p.A8 + ((size_t)(k + p.koff) * ngrp + rg) * 2 * p.S8 * 32 + lane;
  const uint2* B = check_column<NAE, AH>(p, k, h0);
  const int ea = rg * 32 + lane < p.rows ? p.eA[(size_t)(k + p.koff) * p.rows + rg * 32 + lane] : FX_NAN;
  int d[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};  // [h][q]: row 16 h + lg (+ 8 for q >= 2), column 2 lq (+ 1 for odd q)
#pragma unroll 4
  for (int c = 0; c < p.sample; ++c) {
    const int st = (int)((long long)c * p.S8 / p.sample);
    const uint4 a0 = __ldg(A + (size_t)st * 32), a1 = __ldg(A + (size_t)(p.S8 + st) * 32);
    const uint2 b = __ldg(B + (size_t)st * 4);
    mma_u8(d[0], a0, b);
    mma_u8(d[1], a1, b);
  }
  const unsigned rows = __ballot_sync(0xffffffffu, plain_exp(ea)), cols = plain_columns<NAE, AH>(p, k, h0);
  bool low = false;
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = 16 * h + lg + (q >= 2 ? 8 : 0), t = 2 * lq + (q & 1);
      low |= ((rows >> r) & (cols >> t) & 1u) && d[h][q] < p.least;
    }
  return !__any_sync(0xffffffffu, low);
}

// Second pass: all of K and the norms.  The columns (bit t: h0 + t) of this lane's row (32 rg +
// lane) that stay open.
template <int NAE, int AH>
__device__ __forceinline__ unsigned check_whole(const SliceParams& p, int k, int rg, int h0) {
  const int lane = threadIdx.x & 31, ngrp = (p.rows + 31) / 32;
  const uint4* A = p.A8 + ((size_t)(k + p.koff) * ngrp + rg) * 2 * p.S8 * 32 + lane;
  const uint2* B = check_column<NAE, AH>(p, k, h0);
  float s[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}}, qa[4] = {0.0f, 0.0f, 0.0f, 0.0f}, qb = 0.0f;
  for (int c0 = 0; c0 < p.S8; c0 += 512) {  // 512 steps of 32 products below 2^16 fit in 31 bits
    int d[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
    unsigned da[4] = {0, 0, 0, 0}, db = 0;
#pragma unroll 2
    for (int st = c0; st < min(p.S8, c0 + 512); ++st) {
      const uint4 a0 = __ldg(A + (size_t)st * 32), a1 = __ldg(A + (size_t)(p.S8 + st) * 32);
      const uint2 b = __ldg(B + (size_t)st * 4);
      mma_u8(d[0], a0, b);
      mma_u8(d[1], a1, b);
      db = __dp4a(b.x, b.x, __dp4a(b.y, b.y, db));
      da[0] = __dp4a(a0.x, a0.x, __dp4a(a0.y, a0.y, da[0]));
      da[1] = __dp4a(a0.z, a0.z, __dp4a(a0.w, a0.w, da[1]));
      da[2] = __dp4a(a1.x, a1.x, __dp4a(a1.y, a1.y, da[2]));
      da[3] = __dp4a(a1.z, a1.z, __dp4a(a1.w, a1.w, da[3]));
    }
    qb += (float)db;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      qa[q] += (float)da[q];
      s[0][q] += (float)d[0][q];
      s[1][q] += (float)d[1][q];
    }
  }
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    qb += __shfl_xor_sync(0xffffffffu, qb, o);
#pragma unroll
    for (int q = 0; q < 4; ++q) qa[q] += __shfl_xor_sync(0xffffffffu, qa[q], o);
  }
  // from the accumulators' places to a row per lane
  const int quarter = lane >> 3, from = (lane & 7) * 4;  // rows 8 quarter ..
  float a2 = 0.0f;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float v = __shfl_sync(0xffffffffu, qa[q], from);
    if (q == quarter) a2 = v;
  }
  const int row = 32 * rg + lane;
  const bool on = row < p.rows && plain_exp(p.eA[(size_t)(k + p.koff) * p.rows + min(row, p.rows - 1)]);
  const unsigned cols = plain_columns<NAE, AH>(p, k, h0);
  unsigned bits = 0;
#pragma unroll
  for (int t = 0; t < AH; ++t) {
    float ab = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float v = __shfl_sync(0xffffffffu, s[q >> 1][2 * (q & 1) + (t & 1)], from + (t >> 1));
      if (q == quarter) ab = v;
    }
    const float b2 = __shfl_sync(0xffffffffu, qb, t * 4);
    if (on && ((cols >> t) & 1u) && !(ab * ab >= SL_CHECK_M * (a2 + b2) + SL_CHECK_K * (float)p.K)) bits |= 1u << t;
  }
  return bits;
}

// Columns h0 .. h0 + AH - 1 of the 32 rows of a warp in binary64; those in bits (bit j: h0 + j)
// of this lane's row are stored.  All open columns at once, so that an element of u is read for
// up to 4 AH products, and a column's element is fetched and converted by one lane: bound by the
// FP64 pipe.  (Unrolled, the code beside the tile loop cost the 12-column contraction 8 %
// when no sum was open.)  With every x -> band sum open, 512 k / 100 bands / 8^3 x: 2.3 ms
// for that contraction (0.12 with none; the FP64-pipe kernel 1.75), the action 2.5 ms
// (pipe: 3.2).
template <int MODE, int NAE, int AH>
__device__ __forceinline__ void sum_binary64(const SliceParams& p, int k, int row, int h0, unsigned bits) {
  constexpr int NI = 32 / AH;  // a lane holds the column element of one (i, j)
  const int lane = threadIdx.x & 31, li = lane / AH, lj = lane - li * AH, r = min(row, p.rows - 1);
  const int t = h0 + lj, v = t / p.na;
  const double2* u = p.u + (size_t)k * p.uk + (MODE == 1 ? (size_t)r * p.ux : (size_t)r);
  const size_t us = MODE == 1 ? 1 : p.ux;
  const unsigned any = __reduce_or_sync(0xffffffffu, bits);  // columns that no row needs are left out
  double2 z[AH], next = u[0];
#pragma unroll
  for (int j = 0; j < AH; ++j) z[j] = make_double2(0.0, 0.0);
#pragma unroll 1
  for (int i0 = 0; i0 < p.K; i0 += NI) {
    double2 b = make_double2(0.0, 0.0);
    const int i = i0 + li;
    if (li < NI && i < p.K) {
      if (MODE == 1) {
        const size_t o = (size_t)i + (size_t)p.nb * ((size_t)k + (size_t)p.nk * (t - v * p.na));
        const double w = p.allow[o];
        b = make_double2(weigh(p.pr[v * p.vstride + o], w), weigh(p.pi[v * p.vstride + o], w));
      } else {
        b = p.f[((p.bshared ? 0 : (size_t)k) * p.K + i) * NAE + t];
        if (p.ex) {
          const int e = p.ex[(size_t)i * NAE + t];
          b = make_double2(fx_to_double(__double_as_longlong(b.x), e), fx_to_double(__double_as_longlong(b.y), e));
        }
      }
    }
#pragma unroll 1
    for (int q = 0; q < min(NI, p.K - i0); ++q) {
      const double2 a = next;
      next = u[(size_t)min(i0 + q + 1, p.K - 1) * us];
#pragma unroll
      for (int j = 0; j < AH; ++j) {
        if (!((any >> j) & 1u)) continue;
        const double br = __shfl_sync(0xffffffffu, b.x, q * AH + j), bi = __shfl_sync(0xffffffffu, b.y, q * AH + j);
        if (MODE == 1) {
          z[j].x += a.x * br - a.y * bi;
          z[j].y += a.x * bi + a.y * br;
        } else {
          z[j].x += a.x * br + a.y * bi;
          z[j].y += a.x * bi - a.y * br;
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < AH; ++j) {
    if (!((bits >> j) & 1u)) continue;
    if (MODE == 1) {
      p.phi[((size_t)k * p.rows + row) * NAE + h0 + j] = z[j];
    } else {
      const int vj = (h0 + j) / p.na;
      double* out = p.part + (size_t)vj * 2 * p.npsi + (size_t)row +
                    (size_t)p.nb * ((size_t)k + (size_t)p.nk * (h0 + j - vj * p.na));
      out[0] = p.negate ? -z[j].x : z[j].x;
      out[p.npsi] = p.negate ? -z[j].y : z[j].y;
    }
  }
}

// The sums that the second pass leaves open in a warp's row group (quadrant q4) of the tiles
// t0 .. t1 - 1 in left (bit min(t - t0, 63)): the whole sum goes to the first split, zero to the
// others.  The thread that stored the digits' result overwrites it.
template <int MODE, int NAE, int AH>
__device__ __noinline__ void redo_sums(const SliceParams& p, int t0, int t1, unsigned long long left, int q4, int h0) {
#pragma unroll 1
  for (int t = t0; t < t1; ++t) {
    if (!((left >> min(t - t0, 63)) & 1ull)) continue;
    const SliceTile ti = slice_decode<MODE>(p, t);
    const int rg = ti.mt * (SL_ROWS / 32) + q4, row = 32 * rg + (threadIdx.x & 31);
    if (rg * 32 >= p.rows) continue;
    const unsigned open = check_whole<NAE, AH>(p, ti.k, rg, h0);
    if (!__any_sync(0xffffffffu, open != 0)) continue;
    if (ti.sp == 0) {
      sum_binary64<MODE, NAE, AH>(p, ti.k, row, h0, open);
      continue;
    }
    for (int j = 0; j < AH; ++j) {
      if (!((open >> j) & 1u)) continue;
      const int v = (h0 + j) / p.na;
      double* out = p.part + (size_t)ti.sp * p.part_stride + (size_t)v * 2 * p.npsi + (size_t)row +
                    (size_t)p.nb * ((size_t)ti.k + (size_t)p.nk * (h0 + j - v * p.na));
      out[0] = 0.0;
      out[p.npsi] = 0.0;
    }
  }
}

// MODE 1: band -> x (K = re n, im n stacked; B columns carry the signs of the
// complex product).  MODE 2: x -> band (two planes).  C columns per slice and
// MMA, P MMAs (parts) per K step.
template <int MODE, int C, int P>
__global__ void __launch_bounds__(slice_threads(P == 1 ? C / 2 : C), 1) k_slice_gemm(const __grid_constant__ SliceParams p) {
  constexpr int NAE = P == 1 ? C / 2 : C;        // complex columns
  constexpr int NBOX = MODE == 1 ? SL_S : 2 * SL_S;
  constexpr int ND = SL_S * C;                   // digit rows of a part
  constexpr int N = slice_n(C);                  // MMA N
  constexpr int PL = MODE == 2 && P == 1 ? 2 : 1;  // accumulators of their own per plane
  constexpr int DCOLS = P * PL * N;
  constexpr int ACC = 2 * DCOLS <= 512 ? 2 : 1;
  constexpr uint32_t TCOLS = ACC * DCOLS <= 128 ? 128 : (ACC * DCOLS <= 256 ? 256 : 512);
  constexpr uint32_t PROWS = 23 * C;             // 11 empty slices, 12 digit slices
  constexpr uint32_t PITCH = slice_rows(C, P) * 16;  // bytes of a granule of B in shared memory
  constexpr uint32_t IDESC0 = (1u << 4) | ((uint32_t)(SL_ROWS >> 4) << 24);
  extern __shared__ __align__(1024) uint8_t smem[];
  const int S = p.stages;
  const uint32_t slot_bytes = p.KC * PITCH, stage_bytes = p.stage_bytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 2 * slot_bytes + S * stage_bytes);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * SL_MAX_STAGES + 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t b_smem = su32(smem), a_smem = b_smem + 2 * slot_bytes;
  const uint32_t full0 = su32(bars), empty0 = full0 + 8 * SL_MAX_STAGES;
  const uint32_t bfull0 = empty0 + 8 * SL_MAX_STAGES, bempty0 = bfull0 + 16, tfull0 = bempty0 + 16, tempty0 = tfull0 + 16;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int t0 = (int)((long long)p.ntiles * blockIdx.x / gridDim.x);
  const int t1 = (int)((long long)p.ntiles * (blockIdx.x + 1) / gridDim.x);

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bfull0 + 8 * b, 1);
      mbar_init(bempty0 + 8 * b, 1);
      mbar_init(tfull0 + 8 * b, 1);
      mbar_init(tempty0 + 8 * b, (NAE == 4 ? 192 : 320) - 64);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tmem_slot)), "r"(TCOLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  {  // the empty slices of B stay zero; A stages too when an odd granule count leaves one that is never
     // written (it meets zero digits, but must hold finite ones)
    const uint32_t zb = 2 * slot_bytes + ((p.G & 1) ? S * stage_bytes : 0);
    for (uint32_t i = threadIdx.x * 16; i < zb; i += blockDim.x * 16)
      *reinterpret_cast<uint4*>(smem + i) = make_uint4(0, 0, 0, 0);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const bool keepb = p.nch == 1;  // one chunk: B stays while k does

  if (warp == 0) {
    // -------------------------------------------------------------- producer
    uint32_t stage = 0, phase = 0, slot = 0, bphase = 0;
    int armed[SL_MAX_STAGES], barmed[2] = {-1, -1};
#pragma unroll
    for (int s = 0; s < SL_MAX_STAGES; ++s) armed[s] = -1;
    bool ok = true;
    int lastk = -1;
    for (int t = t0; t < t1 && ok && !p.starve; ++t) {
      const SliceTile ti = slice_decode<MODE>(p, t);
      const uint8_t* At = p.A + ((size_t)(ti.k + p.koff) * p.R + (size_t)SL_ROWS * ti.mt) * 16 * p.G * NBOX;
      const uint8_t* Bk = p.B + (p.bshared ? 0 : (size_t)ti.k) * p.Ge * (P * ND * 16);
      for (int c = ti.c0; c < ti.c1 && ok; ++c) {
        const int gc = min(p.KC, p.G - c * p.KC), gce = (gc + 1) & ~1;
        if (!keepb || ti.k != lastk) {
          ok = mbar_wait(bempty0 + 8 * slot, bphase ^ 1, abort_flag, TC_WAIT_CYCLES);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          if (lane == 0) mbar_expect_tx(bfull0 + 8 * slot, (uint32_t)gce * P * ND * 16);
          __syncwarp();
          const uint8_t* src = Bk + (size_t)c * p.KC * (P * ND * 16);
          for (int i = lane; i < gce * P; i += 32)
            bulk_load(b_smem + slot * slot_bytes + (i / P) * PITCH + ((i % P) * PROWS + 11 * C) * 16,
                      src + (size_t)i * (ND * 16), ND * 16, bfull0 + 8 * slot);
          barmed[slot] = (int)bphase;
          slot ^= 1;
          if (slot == 0) bphase ^= 1;
          lastk = ti.k;
        }
        const uint32_t bytes = (uint32_t)gc * ti.rt * 16 * p.sb;
        const uint8_t* src = At + (size_t)c * p.KC * ti.rt * 16 * NBOX;
        for (int b = 0; b < NBOX / p.sb; ++b) {
          ok = mbar_wait(empty0 + 8 * stage, phase ^ 1, abort_flag, TC_WAIT_CYCLES);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          if (lane == 0) {
            mbar_expect_tx(full0 + 8 * stage, bytes);
            bulk_load(a_smem + stage * stage_bytes, src + (size_t)b * bytes, bytes, full0 + 8 * stage);
          }
          armed[stage] = (int)phase;
          if (++stage == (uint32_t)S) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
    if (!ok && lane == 0) {
      *abort_flag = 1;
      atomicOr(p.err, 1);
    }
    // drain: never leave a bulk copy in flight
    for (int s = 0; s < S; ++s)
      if (armed[s] >= 0) {
        const long long w0 = clock64();
        while (!mbar_test(full0 + 8 * s, (uint32_t)armed[s]) && clock64() - w0 < TC_WAIT_CYCLES) {
        }
      }
    for (int s = 0; s < 2; ++s)
      if (barmed[s] >= 0) {
        const long long w0 = clock64();
        while (!mbar_test(bfull0 + 8 * s, (uint32_t)barmed[s]) && clock64() - w0 < TC_WAIT_CYCLES) {
        }
      }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer
    // the whole warp runs the (warp-uniform) loop, one elected lane issues
    uint32_t stage = 0, phase = 0, slot = 0, bphase = 0, acc = 0, acc_phase = 0;
    int last_stage = -1;
    uint32_t last_phase = 0;
    bool ok = true;
    int lastk = -1;
    const bool leader = elect_one();
    for (int t = t0; t < t1 && ok; ++t) {
      const SliceTile ti = slice_decode<MODE>(p, t);
      ok = __all_sync(0xffffffffu, mbar_wait(tempty0 + 8 * acc, acc_phase ^ 1, abort_flag, TC_WAIT_CYCLES));
      if (!ok) break;
      tc_fence_after();
      const uint32_t dt = tmem_base + acc * DCOLS;
      const uint32_t lba = (uint32_t)ti.rt * 16;
      for (int c = ti.c0; c < ti.c1 && ok; ++c) {
        const int gc = min(p.KC, p.G - c * p.KC), steps = (gc + 1) >> 1;
        if (!keepb || ti.k != lastk) {
          ok = __all_sync(0xffffffffu, mbar_wait(bfull0 + 8 * slot, bphase, abort_flag, TC_WAIT_CYCLES));
          if (!ok) break;
          lastk = ti.k;
        }
        for (int b0 = 0; b0 < NBOX; b0 += p.sb) {
          ok = __all_sync(0xffffffffu, mbar_wait(full0 + 8 * stage, phase, abort_flag, TC_WAIT_CYCLES));
          if (!ok) break;
          tc_fence_after();
          for (int b = b0; b < b0 + p.sb; ++b) {
            const int plane = b / SL_S, i = b - plane * SL_S;
            uint32_t ad = plain_desc(a_smem + stage * stage_bytes + (b - b0) * gc * lba, lba);
            // the first i column groups of slice i only meet empty slices: N shrinks in steps of 16
            const uint32_t ni = (uint32_t)(N - i * C + 15) & ~15u, off = N - ni;
            const uint32_t idesc = IDESC0 | ((ni >> 3) << 17);
            uint32_t bd = plain_desc(b_smem + slot * slot_bytes + ((11 - i) * C + off) * 16, PITCH);
            const uint32_t d0 = dt + (PL == 2 ? plane * N : 0) + off;
            // the first MMA of an accumulator overwrites it
            uint32_t accum = (c > ti.c0 || (PL == 2 ? i > 0 : b > 0)) ? 1u : 0u;
            if (leader) {
#pragma unroll 4
              for (int g = 0; g < steps; ++g) {
#pragma unroll
                for (int q = 0; q < P; ++q) {
                  const uint32_t part = MODE == 2 ? (uint32_t)(q ^ plane) : (uint32_t)q;  // im plane: parts swapped
                  const uint32_t neg = (MODE == 2 && P == 2 && q == 1 && plane == 1) ? (1u << 13) : 0u;
                  umma_fp8(d0 + q * N, ad, bd + (P == 2 ? part * PROWS : 0u), idesc | neg, accum);
                }
                accum = 1u;
                ad += 2 * (lba >> 4);
                bd += 2 * (PITCH >> 4);
              }
            }
          }
          if (leader) umma_commit(empty0 + 8 * stage);
          __syncwarp();
          last_stage = (int)stage;
          last_phase = phase;
          if (++stage == (uint32_t)S) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        if (!keepb || t + 1 == t1 || slice_decode<MODE>(p, t + 1).k != ti.k) {
          if (leader) umma_commit(bempty0 + 8 * slot);
          slot ^= 1;
          if (slot == 0) bphase ^= 1;
        }
      }
      if (!ok) break;
      if (leader) umma_commit(tfull0 + 8 * acc);
      if (ACC == 2) acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
    if (!ok && leader) {
      *abort_flag = 1;
      atomicOr(p.err, 2);
    }
    if (last_stage >= 0) {  // drain: every issued MMA finished reading shared memory
      const long long w0 = clock64();
      while (!mbar_test(empty0 + 8 * last_stage, last_phase) && clock64() - w0 < TC_WAIT_CYCLES) {
      }
    }
  } else {
    // -------------------------------------------------------------- epilogue
    constexpr int AH = NAE == 4 ? 4 : NAE / 2;       // columns of a thread
    constexpr uint32_t PART = P == 1 ? NAE : N;      // accumulator columns between the parts
    const int q4 = warp & 3;  // tensor-memory lane quadrant of this warp
    const int row = q4 * 32 + lane, h0 = ((warp - 2) >> 2) * AH;
    uint32_t acc = 0, acc_phase = 0;
    unsigned long long left = 0;  // tiles that the first pass of the check does not clear, see redo_sums
    for (int t = t0; t < t1; ++t) {
      const SliceTile ti = slice_decode<MODE>(p, t);
      __syncwarp();
      if (!check_part<NAE, AH>(p, ti.k, ti.mt * (SL_ROWS / 32) + q4, h0)) left |= 1ull << min(t - t0, 63);
      // every lane the same way: the loop's warp-wide steps need all of them
      if (!__all_sync(0xffffffffu, mbar_wait(tfull0 + 8 * acc, acc_phase, abort_flag, TC_WAIT_CYCLES))) {
        *abort_flag = 1;
        atomicOr(p.err, 4);
        left = 0;
        break;
      }
      tc_fence_after();
      const uint32_t ta = tmem_base + ((uint32_t)(q4 * 32) << 16) + acc * DCOLS + h0;
      long long hi[2][AH], lo[2][AH];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        add_groups<AH, C, 7>(ta + q * PART, hi[q]);
        add_groups<AH, C, 6>(ta + q * PART + 7 * C, lo[q]);
      }
      if (PL == 2) {  // out = (re plane) phi' - i (im plane) phi'
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          long long im[AH];
          add_groups<AH, C, 7>(ta + N + (1 - q) * PART, im);
#pragma unroll
          for (int a = 0; a < AH; ++a) hi[q][a] += q ? -im[a] : im[a];
          add_groups<AH, C, 6>(ta + N + (1 - q) * PART + 7 * C, im);
#pragma unroll
          for (int a = 0; a < AH; ++a) lo[q][a] += q ? -im[a] : im[a];
        }
      }
      tc_fence_before();
      mbar_arrive(tempty0 + 8 * acc);
      if (ACC == 2) acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
      const int r = ti.mt * SL_ROWS + row;
      if (r < p.rows) {
        const int ea = p.eA[(size_t)(ti.k + p.koff) * p.rows + r];
        const int* eb = p.eB + (p.bshared ? 0 : (size_t)ti.k) * NAE;
#pragma unroll
        for (int j = 0; j < AH; ++j) {
          const int a = h0 + j;
          if (p.spin >= 0 && (a & 1) != p.spin) continue;
          const int e = eb[a];
          const int es = ea + e - 2 * SL_FRAC + 50;
          double vr = fx_to_double(hi[0][j], lo[0][j], es);
          double vi = fx_to_double(hi[1][j], lo[1][j], es);
          if (ea == FX_NAN || e == FX_NAN) vr = vi = __longlong_as_double(0x7ff8000000000000ll);
          if (MODE == 1) {
            p.phi[((size_t)ti.k * p.rows + r) * NAE + a] = make_double2(vr, vi);
          } else {
            const int v = a / p.na;
            double* out = p.part + (size_t)ti.sp * p.part_stride + (size_t)v * 2 * p.npsi;
            const size_t idx = (size_t)r + (size_t)p.nb * ((size_t)ti.k + (size_t)p.nk * (a - v * p.na));
            out[idx] = p.negate ? -vr : vr;
            out[p.npsi + idx] = p.negate ? -vi : vi;
          }
        }
      }
    }
    // sums that the digits do not hold as well as binary64 (after the loop, out of the pipeline's waits)
    if (left) redo_sums<MODE, NAE, AH>(p, t0, t1, left, q4, h0);
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TCOLS) : "memory");
  }
}

// ------------------------------------------------------------- digit operands

// biased fixed point: the 60-bit integer plus 16 in every base-32 digit
__device__ __forceinline__ unsigned long long fix_point(double v, int e) {
  return SL_BIAS + (unsigned long long)fx_from<SL_FRAC>(v, e);
}
// digit s (0 most significant) of a biased fixed-point value as an exact float
__device__ __forceinline__ float digit_of(unsigned long long t, int s) {
  unsigned r = (unsigned)(t >> (5 * (SL_S - 1 - s)));
  if (s) r &= 31u;
  return __int_as_float((int)(0x4B000000u | r)) - 8388624.0f;
}
__device__ __forceinline__ unsigned fp8x4(float a, float b, float c, float d) {
  unsigned short lo, hi;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(lo) : "f"(b), "f"(a));
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(hi) : "f"(d), "f"(c));
  return (unsigned)lo | ((unsigned)hi << 16);
}
__device__ __forceinline__ unsigned digits4(const unsigned long long* t, int s) {
  return fp8x4(digit_of(t[0], s), digit_of(t[1], s), digit_of(t[2], s), digit_of(t[3], s));
}
__device__ __forceinline__ uint4 digits16(const unsigned long long* t, int s) {
  return make_uint4(digits4(t, s), digits4(t + 4, s), digits4(t + 8, s), digits4(t + 12, s));
}

// Row exponents of the band -> x operand: rows (k, x), over n.  One warp per row.
// src: element (x, k, n) at x*sx + k*sk + n.
__global__ void k_slice_exp_rows(const double2* __restrict__ u, size_t sx, size_t sk, int nb, int nk, int nx,
                                 int* __restrict__ e) {
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= (long long)nk * nx) return;
  const int k = (int)(w / nx), x = (int)(w % nx);
  const double2* r = u + x * sx + k * sk;
  unsigned m = 0;
  for (int n = lane; n < nb; n += 32) m = max(m, max(fx_mag(r[n].x), fx_mag(r[n].y)));
  m = __reduce_max_sync(0xffffffffu, m);
  if (lane == 0) e[w] = fx_exp(m);
}

// Row exponents of the x -> band operand: rows (k, n), over x.  Block (32 n, 8).
__global__ void k_slice_exp_cols(const double2* __restrict__ u, size_t sx, size_t sk, int nb, int nk, int nx,
                                 int* __restrict__ e) {
  __shared__ unsigned sh[8][32];
  const int n = blockIdx.x * 32 + threadIdx.x, k = blockIdx.y;
  unsigned m = 0;
  if (n < nb)
    for (int x = threadIdx.y; x < nx; x += 8) {
      const double2 v = u[x * sx + k * sk + n];
      m = max(m, max(fx_mag(v.x), fx_mag(v.y)));
    }
  sh[threadIdx.y][threadIdx.x] = m;
  __syncthreads();
  if (threadIdx.y == 0 && n < nb) {
    for (int i = 1; i < 8; ++i) m = max(m, sh[i][threadIdx.x]);
    e[(size_t)k * nb + n] = fx_exp(m);
  }
}

// Where 16 digit bytes of (k, row, box, granule) go (see the file comment).
__device__ __forceinline__ size_t slice_a_off(const SliceParams& p, int nbox, int k, int row, int box, int g) {
  const int mt = row / SL_ROWS, rt = mt == p.nt - 1 ? p.rl : SL_ROWS;
  const int c = g / p.KC, gc = min(p.KC, p.G - c * p.KC);
  return ((size_t)k * p.R + (size_t)SL_ROWS * mt) * 16 * p.G * nbox +
         ((size_t)c * p.KC * nbox + (size_t)box * gc + (g - c * p.KC)) * rt * 16 + (size_t)(row - mt * SL_ROWS) * 16;
}

// Digits of the band -> x operand; one thread per (k, granule, row), rows fastest.
__global__ void k_slice_build_rows(const double2* __restrict__ u, size_t sx, size_t sk, int nb, const SliceParams p,
                                   const int* __restrict__ e, uint8_t* __restrict__ A, int koff) {
  const long long tot = (long long)p.nk * p.G * p.R;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < tot; i += (long long)gridDim.x * blockDim.x) {
    const int row = (int)(i % p.R);
    const int g = (int)((i / p.R) % p.G), k = (int)(i / ((long long)p.R * p.G));
    unsigned long long t[16];
    const bool in = row < p.rows;
    const int er = in ? e[(size_t)k * p.rows + row] : 0;
    const double2* r = u + (size_t)row * sx + (size_t)k * sk;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int K = 16 * g + j, n = K < nb ? K : K - nb;
      t[j] = SL_BIAS;
      if (in && K < 2 * nb) t[j] = fix_point(K < nb ? r[n].x : r[n].y, er);
    }
#pragma unroll 1
    for (int s = 0; s < SL_S; ++s)
      *reinterpret_cast<uint4*>(A + slice_a_off(p, SL_S, k + koff, row, s, g)) = digits16(t, s);
  }
}

// Digits of the x -> band operand; one thread per (k, plane, granule of x, row n), rows fastest.
__global__ void k_slice_build_cols(const double2* __restrict__ u, size_t sx, size_t sk, int nx, const SliceParams p,
                                   const int* __restrict__ e, uint8_t* __restrict__ A, int koff) {
  const long long tot = (long long)p.nk * 2 * p.G * p.R;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < tot; i += (long long)gridDim.x * blockDim.x) {
    const int n = (int)(i % p.R);
    const long long q = i / p.R;
    const int g = (int)(q % p.G), plane = (int)((q / p.G) & 1), k = (int)(q / (2 * p.G));
    unsigned long long t[16];
    const bool in = n < p.rows;
    const int er = in ? e[(size_t)k * p.rows + n] : 0;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int x = 16 * g + j;
      t[j] = SL_BIAS;
      if (in && x < nx) {
        const double2 v = u[(size_t)x * sx + (size_t)k * sk + n];
        t[j] = fix_point(plane ? v.y : v.x, er);
      }
    }
#pragma unroll 1
    for (int s = 0; s < SL_S; ++s)
      *reinterpret_cast<uint4*>(A + slice_a_off(p, 2 * SL_S, k + koff, n, plane * SL_S + s, g)) = digits16(t, s);
  }
}

// 8-bit magnitude of a complex element against its block exponent, rounded down: the larger
// part is at least m 2^(e - 8).
__device__ __forceinline__ unsigned mag8(long long re, long long im) {
  const long long a = max(re < 0 ? -re : re, im < 0 ? -im : im);
  return min((unsigned)(a >> (SL_FRAC - 8)), 255u);
}
__device__ __forceinline__ unsigned mag8(double re, double im, int e) {
  return mag8(fx_from<SL_FRAC>(re, e), fx_from<SL_FRAC>(im, e));
}

// psi operand of one k-point per CTA: q = allow o psi of nae columns t = (vector,
// channel); column exponents, then digits of
//   part 0 (Re phi): K = (re n) -> qr, (im n) -> -qi;  part 1 (Im phi): (re n) -> qi, (im n) -> qr.
// merged: row order [slice][part][t], else [part][slice][t].  M: magnitudes [k][t][32 S8].
// Clears the maxima that the k-mesh transform of this action collects.
__global__ void __launch_bounds__(256)
    k_slice_prep_b1(const double* __restrict__ pr, const double* __restrict__ pi, size_t vstride,
                    const double* __restrict__ allow, int nb, int nk, int na, int nae, int Ge, int merged,
                    uint8_t* __restrict__ B, int* __restrict__ eB, int* __restrict__ mx, uint8_t* __restrict__ M, int S8) {
  __shared__ int se[OCN_MAX_NA];
  const int k = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if ((int)threadIdx.x < nae) mx[(size_t)k * nae + threadIdx.x] = -FX_NAN;
  for (int t = warp; t < nae; t += 8) {
    const int v = t / na, a = t - v * na;
    const size_t base = (size_t)nb * ((size_t)k + (size_t)nk * a);
    unsigned m = 0;
    for (int n = lane; n < nb; n += 32) {
      const double w = allow[base + n];
      m = max(m, max(fx_mag(weigh(pr[v * vstride + base + n], w)), fx_mag(weigh(pi[v * vstride + base + n], w))));
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) {
      se[t] = fx_exp(m);
      eB[(size_t)k * nae + t] = se[t];
    }
  }
  __syncthreads();
  const int items = Ge * 2 * nae * 4;
  for (int i = threadIdx.x; i < items; i += blockDim.x) {
    const int qd = i & 3, r = i >> 2;
    const int t = r % nae, part = (r / nae) & 1, g = r / (2 * nae);
    const int v = t / na, a = t - v * na, e = se[t];
    const size_t base = (size_t)nb * ((size_t)k + (size_t)nk * a);
    unsigned long long f[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int K = 16 * g + 4 * qd + j, c = K >= nb, n = c ? K - nb : K;
      f[j] = SL_BIAS;
      if (K < 2 * nb) {
        const double w = allow[base + n];
        const double x = weigh(((part ^ c) ? pi : pr)[v * vstride + base + n], w);
        f[j] = fix_point(part == 0 && c ? -x : x, e);
      }
    }
    uint8_t* out = B + ((size_t)k * Ge + g) * 2 * SL_S * nae * 16 + 4 * qd;
#pragma unroll 1
    for (int s = 0; s < SL_S; ++s) {
      const int row = merged ? (s * 2 + part) * nae + t : (part * SL_S + s) * nae + t;
      *reinterpret_cast<unsigned*>(out + (size_t)row * 16) = digits4(f, s);
    }
  }
  for (int i = threadIdx.x; i < nae * S8 * 8; i += blockDim.x) {
    const int t = i / (8 * S8), n0 = 4 * (i - t * 8 * S8), v = t / na, a = t - v * na;
    const size_t base = (size_t)nb * ((size_t)k + (size_t)nk * a);
    unsigned m = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + j;
      if (n >= nb) break;
      const double w = allow[base + n];
      m |= mag8(weigh(pr[v * vstride + base + n], w), weigh(pi[v * vstride + base + n], w), se[t]) << (8 * j);
    }
    *reinterpret_cast<unsigned*>(M + ((size_t)k * nae + t) * 32 * S8 + n0) = m;
  }
}

// Exponent maxima mx[k][t] of src[k*nx + x][t] (operands that do not come from the
// fixed-point k-mesh transform).
__global__ void __launch_bounds__(512)
    k_slice_col_max(const double2* __restrict__ src, int nx, int nae, int* __restrict__ mx) {
  __shared__ unsigned sm[OCN_MAX_NA];
  const int k = blockIdx.x;
  if (threadIdx.x < OCN_MAX_NA) sm[threadIdx.x] = 0;
  __syncthreads();
  const double2* f = src + (size_t)k * nx * nae;
  const int step = (int)blockDim.x / nae * nae;  // a multiple of nae: a thread's column is fixed
  if ((int)threadIdx.x < step) {
    unsigned m = 0;
    for (int i = threadIdx.x; i < nx * nae; i += step) m = max(m, max(fx_mag(f[i].x), fx_mag(f[i].y)));
    atomicMax(&sm[threadIdx.x % nae], m);
  }
  __syncthreads();
  if ((int)threadIdx.x < nae) mx[(size_t)k * nae + threadIdx.x] = fx_exp(sm[threadIdx.x]);
}

// int 2^s rounded to nearest, plus the digit bias; |int 2^s| <= 2^59
__device__ __forceinline__ unsigned long long fix_int(long long v, int s) {
  if (s >= 0) return SL_BIAS + ((unsigned long long)v << s);
  const int r = min(-s, 63);
  return SL_BIAS + (unsigned long long)((v + (1ll << (r - 1))) >> r);
}

// phi' operand from src[k*nx + x][t] (parts: re, im) and its column exponents: digits,
// rows and M as k_slice_prep_b1.  INT: src holds integers with exponents ex[x][t], else
// binary64.  grid (ceil(items / block), Nk); a thread makes four x of one column, both
// parts (reads 64-byte runs, writes 4-byte words of 64-byte runs).
template <bool INT>
__global__ void __launch_bounds__(256)
    k_slice_prep_b2(const double2* __restrict__ src, const int* __restrict__ ex, int nx, int nae, int Ge, int merged,
                    const int* __restrict__ mx, uint8_t* __restrict__ B, int* __restrict__ eB, uint8_t* __restrict__ M,
                    int S8) {
  const int k = blockIdx.y;
  if (blockIdx.x == 0 && (int)threadIdx.x < nae)
    eB[(size_t)k * nae + threadIdx.x] = mx[(size_t)k * nae + threadIdx.x];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= Ge * nae * 4) return;
  const int qd = i & 3, r = i >> 2;
  const int t = r % nae, g = r / nae, e = mx[(size_t)k * nae + t];
  const double2* f = src + (size_t)k * nx * nae + t;
  unsigned long long fr[4], fi[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int x = 16 * g + 4 * qd + j;
    fr[j] = fi[j] = SL_BIAS;
    if (x < nx) {
      if constexpr (INT) {
        const longlong2 v = reinterpret_cast<const longlong2*>(f)[(size_t)x * nae];
        if (e < FX_NAN) {
          const int s = ex[(size_t)x * nae + t] + SL_FRAC - e;
          fr[j] = fix_int(v.x, s);
          fi[j] = fix_int(v.y, s);
        }
      } else {
        const double2 v = f[(size_t)x * nae];
        fr[j] = fix_point(v.x, e);
        fi[j] = fix_point(v.y, e);
      }
    }
  }
  uint8_t* out = B + ((size_t)k * Ge + g) * 2 * SL_S * nae * 16 + (size_t)t * 16 + 4 * qd;
#pragma unroll 4
  for (int s = 0; s < SL_S; ++s) {
    *reinterpret_cast<unsigned*>(out + (size_t)(merged ? 2 * s : s) * nae * 16) = digits4(fr, s);
    *reinterpret_cast<unsigned*>(out + (size_t)(merged ? 2 * s + 1 : SL_S + s) * nae * 16) = digits4(fi, s);
  }
  {
    unsigned m = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) m |= mag8((long long)(fr[j] - SL_BIAS), (long long)(fi[j] - SL_BIAS)) << (8 * j);
    *reinterpret_cast<unsigned*>(M + ((size_t)k * nae + t) * 32 * S8 + 16 * g + 4 * qd) = m;
  }
}

// Magnitudes of the u operand in the order in which check_part's lanes hold them, [spin k]
// [group of 32 rows][half][32 K][lane][16 bytes]: lane 4 g + q has K = 8 q .. 8 q + 7 of rows g
// and g + 8 of its half.  One thread per 16 bytes.  MODE 1: rows x over n; MODE 2: rows n over x.
template <int MODE>
__global__ void k_slice_build_mag(const double2* __restrict__ u, size_t sx, size_t sk, int nk, int rows, int K,
                                  const int* __restrict__ e, uint4* __restrict__ M, int koff) {
  const int ngrp = (rows + 31) / 32, S = (K + 31) / 32;
  const long long tot = (long long)nk * ngrp * 2 * S * 32;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < tot; i += (long long)gridDim.x * blockDim.x) {
    const int lane = (int)(i & 31), st = (int)((i >> 5) % S);
    const long long h = (i >> 5) / S;  // (k ngrp + group) 2 + half
    const int k = (int)(h / (2 * ngrp)), row0 = (int)(h % (2 * ngrp)) * 16 + (lane >> 2);
    unsigned w[4] = {0, 0, 0, 0};
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int row = row0 + (j >= 8 ? 8 : 0), c = 32 * st + 8 * (lane & 3) + (j & 7);
      if (row >= rows || c >= K) continue;
      const double2 v = MODE == 1 ? u[(size_t)row * sx + (size_t)k * sk + c] : u[(size_t)c * sx + (size_t)k * sk + row];
      w[j >> 2] |= mag8(v.x, v.y, e[(size_t)k * rows + row]) << (8 * (j & 3));
    }
    M[((size_t)koff * ngrp * 2 * S) * 32 + i] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// amp[i] = sum_k part[k][i], i < n (OCEAN_multiplet.f90:1730-1783's sum over k): a CTA
// owns 32 outputs, its 16 warps take every 16th k, warp 0 adds the partials in order.
__global__ void __launch_bounds__(512)
    k_slice_amp_reduce(const double2* __restrict__ part, double2* __restrict__ amp, int nk, int n) {
  __shared__ double2 sh[16][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
  double2 s = make_double2(0.0, 0.0);
  if (i < n)
    for (int k = w; k < nk; k += 16) {
      const double2 v = part[(size_t)k * n + i];
      s.x += v.x;
      s.y += v.y;
    }
  sh[w][lane] = s;
  __syncthreads();
  if (w == 0 && i < n) {
    for (int g = 1; g < 16; ++g) {
      s.x += sh[g][lane].x;
      s.y += sh[g][lane].y;
    }
    amp[i] = s;
  }
}

typedef void (*SliceFn)(const SliceParams);
SliceFn slice_fn(int mode, int nae) {
  if (mode == 1) return nae == 4 ? k_slice_gemm<1, 8, 1> : (nae == 8 ? k_slice_gemm<1, 16, 1> : k_slice_gemm<1, 12, 2>);
  return nae == 4 ? k_slice_gemm<2, 8, 1> : (nae == 8 ? k_slice_gemm<2, 16, 1> : k_slice_gemm<2, 12, 2>);
}
inline bool slice_merged(int nae) { return nae <= 8; }
// bytes of a granule of B in shared memory
size_t slice_pitch(int nae) {
  const int C = slice_merged(nae) ? 2 * nae : nae, P = slice_merged(nae) ? 1 : 2;
  return (size_t)slice_rows(C, P) * 16;
}

// One contraction: geometry, operand A (digits and exponents) and launch shape.
struct SliceGemm {
  SliceParams p{};
  uint8_t* A = nullptr;
  uint8_t* A8 = nullptr;     // magnitudes (k_slice_build_mag)
  int* eA = nullptr;
  int mode = 1, nbox = SL_S, nae = 4, grid = 1;
  int K = 1;                 // complex products of a sum
  size_t smem = 0;
  size_t a_bytes(int spins) const { return (size_t)spins * p.nk * p.R * 16 * p.G * nbox; }
  int s8() const { return (K + 31) / 32; }  // steps of 32 K of the magnitudes
  size_t a8_bytes(int spins) const { return (size_t)spins * p.nk * ((p.rows + 31) / 32) * 32 * 32 * s8(); }
  size_t b8_bytes() const { return (size_t)(p.bshared ? 1 : p.nk) * nae * 32 * s8(); }
  size_t b_bytes() const { return (size_t)(p.bshared ? 1 : p.nk) * p.Ge * 2 * SL_S * nae * 16; }
};

// rows and summed index of a contraction of nae columns (K complex products, stacked as re
// and im for band -> x); the largest K chunk whose
// two B slots and at least four A stages fit in shared memory (16 granules at most
// for one resident B operand, 12 for streamed ones) with the widest columns, nae_max,
// that share the A operand: its order depends on the chunks.
void slice_plan(SliceGemm* s, int mode, int nae, int nae_max, int nk, int rows, int K, int sm_count,
                double cost_split) {
  SliceParams& p = s->p;
  s->mode = mode;
  s->nae = nae;
  s->nbox = mode == 1 ? SL_S : 2 * SL_S;
  s->K = K;
  if (mode == 1) K *= 2;
  p.nk = nk;
  p.rows = rows;
  p.nt = (rows + SL_ROWS - 1) / SL_ROWS;
  p.rl = (rows - (p.nt - 1) * SL_ROWS + 7) / 8 * 8;
  p.R = (p.nt - 1) * SL_ROWS + p.rl;
  p.G = (K + 15) / 16;
  p.Ge = (p.G + 1) & ~1;
  const size_t pitch = slice_pitch(nae), pitch_max = slice_pitch(nae_max);
  const int cap = mode == 1 ? 16 : 12;
  int kc = std::min(cap, p.Ge);
  while (kc > 2 && kc * (2 * pitch_max + 4 * SL_ROWS * 16) > SL_SMEM) kc -= 2;
  p.KC = kc;
  p.ks = 1;
  if (mode == 2) {
    // K chunk and splits: the least modelled time of the busiest SM's share of A at
    // 45 GB/s per SM, 0.6 us per chunk and the partial sums' round trip (cost_split
    // seconds per slice); a smaller chunk or another split has to gain 3% (1s case of
    // 512 k / 100 bands: 12 granules in 3 splits 358 us, 6 in 2 splits 371 us; 64 k /
    // 32 bands: 12 in 2 splits 22 us, 8 in 2 splits 18 us).  K per accumulation
    // stays within the exact range.
    const double a_gran = (double)(p.nt > 1 ? SL_ROWS : p.rl) * 16 * s->nbox / 45e9;
    double best = 1e30;
    for (int q = kc; q >= std::min(kc, 4); q -= 2) {
      const int nch = (p.G + q - 1) / q, most = SL_MAX_K / (16 * q), least = (nch + most - 1) / most;
      for (int r = least; r <= std::max(least, std::min(nch, 8)); ++r) {
        const int cps = (nch + r - 1) / r, ks = (nch + cps - 1) / cps;
        const long long tiles = (long long)nk * p.nt * ks;
        const double waves = (double)((tiles + sm_count - 1) / sm_count);
        const double t = waves * (std::min(cps * q, p.G) * a_gran + cps * 0.6e-6) + ks * cost_split;
        if (t < 0.97 * best) {
          best = t;
          p.KC = q;
          p.ks = ks;
        }
      }
    }
  }
  p.nch = (p.G + p.KC - 1) / p.KC;
  p.cps = (p.nch + p.ks - 1) / p.ks;
  // boxes per stage: up to 32 KB in one copy and one wait (short rows or few granules
  // make small boxes), with four stages at least.  An MMA reads 128 rows: behind the
  // last box of a tile of fewer rows that runs past the data by up to 127 rows.
  const int rt = p.nt > 1 ? SL_ROWS : p.rl;
  const size_t box = (size_t)p.KC * rt * 16, room = SL_SMEM - 2 * p.KC * pitch;
  for (int sb : {12, 6, 4, 3, 2, 1}) {
    p.sb = sb;
    p.stage_bytes = (uint32_t)((sb * box + (size_t)(SL_ROWS - rt) * 16 + 127) / 128 * 128);
    if (sb == 1 || (sb * box <= 32 * 1024 && 4 * (size_t)p.stage_bytes <= room)) break;
  }
  p.stages = (int)std::min<size_t>(SL_MAX_STAGES, room / p.stage_bytes);
  s->smem = 2 * p.KC * pitch + (size_t)p.stages * p.stage_bytes + 256;  // + barriers
  p.ntiles = nk * p.nt * p.ks;
  p.spin = -1;
  s->grid = std::min(p.ntiles, sm_count);
}

}  // namespace

struct SliceLR {
  bool ready = false;
  int nvs = 1;             // most vectors per launch (12 columns)
  SliceGemm g1[3], g2[3];  // band -> x, x -> band of 1, 2, 3 vectors; A is held by [0] and shared
  uint8_t *b1 = nullptr, *b2 = nullptr;
  uint8_t *m1 = nullptr, *m2 = nullptr;  // magnitudes of the columns
  int *e1 = nullptr, *e2 = nullptr;
  int* mx2 = nullptr;      // exponent maxima of phi' per (k, column)
  int* ex2 = nullptr;      // exponents of phi' per (x, column)
  // multiplet projectors (fg_combo): amplitudes and back-projection
  bool mult_ready = false;
  SliceGemm gm1, gm2;
  uint8_t* bm = nullptr;
  uint8_t* mm = nullptr;
  int* em = nullptr;
  int* mxm = nullptr;
  double2* amp_part = nullptr;  // [k][p][a]
  int* d_err = nullptr;
  int starve = 0;
};

namespace {

template <typename T>
int salloc(ocn_ctx* c, T** p, size_t n) {
  cudaError_t e = cudaMalloc(reinterpret_cast<void**>(p), n * sizeof(T));
  if (e != cudaSuccess) return set_err(c, OCN_ERR_ALLOC, std::string("cudaMalloc: ") + cudaGetErrorString(e));
  return OCN_OK;
}

void slice_drop_a(ocn_ctx* c) {
  SliceLR* s = c->slice;
  for (SliceGemm* g : {&s->g1[0], &s->g2[0]}) {
    if (g->A) cudaFree(g->A);
    if (g->A8) cudaFree(g->A8);
    if (g->eA) cudaFree(g->eA);
    g->A = g->A8 = nullptr;
    g->eA = nullptr;
  }
  s->ready = false;
  c->lr_xsplit = c->lr_xsplit_pipe;
}

void slice_drop_mult(ocn_ctx* c) {
  SliceLR* s = c->slice;
  for (SliceGemm* g : {&s->gm1, &s->gm2}) {
    if (g->A) cudaFree(g->A);
    if (g->A8) cudaFree(g->A8);
    if (g->eA) cudaFree(g->eA);
    g->A = g->A8 = nullptr;
    g->eA = nullptr;
  }
  for (void* q : {(void*)s->bm, (void*)s->mm, (void*)s->em, (void*)s->mxm, (void*)s->amp_part})
    if (q) cudaFree(q);
  s->bm = s->mm = nullptr;
  s->em = nullptr;
  s->mxm = nullptr;
  s->amp_part = nullptr;
  s->mult_ready = false;
  c->mult_parts = 0;
}

// Digits and exponents of both operands of one spin from src (element (x, k, n) at x*sx + k*sk + n).
int slice_build(ocn_ctx* c, const double2* src, size_t sx, size_t sk, int nx, const SliceGemm& g1, const SliceGemm& g2,
                int spin) {
  const int nk = c->nk, nb = c->nb, blocks = 16 * c->sm_count;
  int* e1 = g1.eA + (size_t)spin * nk * nx;
  int* e2 = g2.eA + (size_t)spin * nk * nb;
  const long long warps = (long long)nk * nx;
  k_slice_exp_rows<<<(unsigned)((warps + 7) / 8), 256, 0, c->stream>>>(src, sx, sk, nb, nk, nx, e1);
  k_slice_build_rows<<<blocks, 256, 0, c->stream>>>(src, sx, sk, nb, g1.p, e1, g1.A, spin * nk);
  k_slice_exp_cols<<<dim3((nb + 31) / 32, nk), dim3(32, 8), 0, c->stream>>>(src, sx, sk, nb, nk, nx, e2);
  k_slice_build_cols<<<blocks, 256, 0, c->stream>>>(src, sx, sk, nx, g2.p, e2, g2.A, spin * nk);
  k_slice_build_mag<1><<<blocks, 256, 0, c->stream>>>(src, sx, sk, nk, nx, nb, e1, reinterpret_cast<uint4*>(g1.A8), spin * nk);
  k_slice_build_mag<2><<<blocks, 256, 0, c->stream>>>(src, sx, sk, nk, nb, nx, e2, reinterpret_cast<uint4*>(g2.A8), spin * nk);
  c->launches += 6;
  OCN_CUDA(c, cudaGetLastError());
  return OCN_OK;
}

// Allocates the A operands of both contractions; false (nothing kept) when they
// would take more than a quarter of the free device memory.
bool slice_alloc_a(ocn_ctx* c, SliceGemm* g1, SliceGemm* g2, int nx) {
  const int ns = c->nspn;
  size_t fr = 0, tot = 0;
  if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) return false;
  if (g1->a_bytes(ns) + g2->a_bytes(ns) + g1->a8_bytes(ns) + g2->a8_bytes(ns) > fr / 4) return false;
  if (salloc(c, &g1->A, g1->a_bytes(ns)) || salloc(c, &g2->A, g2->a_bytes(ns)) ||
      salloc(c, &g1->A8, g1->a8_bytes(ns)) || salloc(c, &g2->A8, g2->a8_bytes(ns)) ||
      salloc(c, &g1->eA, (size_t)ns * c->nk * nx) || salloc(c, &g2->eA, (size_t)ns * c->nk * c->nb)) {
    (void)cudaGetLastError();
    c->err.clear();
    return false;
  }
  return true;
}

// Where the columns of a contraction come from: psi (band -> x) or f (x -> band).
struct SliceColumns {
  const double *pr = nullptr, *pi = nullptr;
  size_t vstride = 0;
  const double2* f = nullptr;
  const int* ex = nullptr;
};

// The contraction of both spins.  g: the launch's geometry, a: the holder of its A operand; B,
// M, eB: the columns' digits, magnitudes and exponents; u: element (spin, x, k, n) at
// spin*us + x*ux + k*uk + n, what the digits of a were built from.
int slice_contract(ocn_ctx* c, const SliceGemm& g, const SliceGemm& a, const uint8_t* B, const uint8_t* M, const int* eB,
                   const SliceColumns& col, const double2* u, size_t us, size_t ux, size_t uk, double2* phi, double* part) {
  SliceParams p = g.p;
  p.A = a.A;
  p.eA = a.eA;
  p.B = B;
  p.eB = eB;
  p.phi = phi;
  p.part = part;
  p.part_stride = c->part_stride;
  p.npsi = c->npsi;
  p.na = c->na;
  p.nb = c->nb;
  p.err = c->slice->d_err;
  p.negate = p.bshared ? 0 : 1;
  p.starve = c->slice->starve;
  p.A8 = reinterpret_cast<const uint4*>(a.A8);
  p.B8 = reinterpret_cast<const uint2*>(M);
  p.K = g.K;
  p.S8 = g.s8();
  const double rk = std::sqrt((double)g.K);
  // ungraded rows: ten times the least sum; at most what 31 bits hold
  p.sample = std::min({p.S8, 512, (int)std::ceil(6.0 * rk / 32.0)});
  p.least = (int)std::ceil(std::sqrt(2.0 * SL_CHECK_M * 255.0 * 255.0 + SL_CHECK_K) * rk);
  p.ux = ux;
  p.uk = uk;
  p.pr = col.pr;
  p.pi = col.pi;
  p.allow = c->d_allow;
  p.vstride = col.vstride;
  p.f = col.f;
  p.ex = col.ex;
  for (int sp = 0; sp < c->nspn; ++sp) {
    p.koff = sp * p.nk;
    p.spin = c->nspn == 2 ? sp : -1;
    p.u = u + sp * us;
    slice_fn(g.mode, g.nae)<<<g.grid, slice_threads(g.nae), g.smem, c->stream>>>(p);
    ++c->launches;
    OCN_CUDA(c, cudaGetLastError());
  }
  return OCN_OK;
}

}  // namespace

// Geometry and vector-side buffers (before ocn_ctx_create sizes the partial sums).
int slice_init(ocn_ctx* c) {
  SliceLR* s = new (std::nothrow) SliceLR();
  if (!s) return set_err(c, OCN_ERR_ALLOC, "host allocation failed");
  c->slice = s;
  s->nvs = std::max(1, std::min(c->nvec, 12 / c->na));
  int rc;
  for (int w = 1; w <= s->nvs; ++w) {
    const int nae = w * c->na, most = s->nvs * c->na;
    const double cost = 32.0 * c->npsi / 6e12;  // the same splits for every width of this context: results do not depend on it
    slice_plan(&s->g1[w - 1], 1, nae, most, c->nk, c->nx, c->nb, c->sm_count, 0.0);
    slice_plan(&s->g2[w - 1], 2, nae, most, c->nk, c->nb, c->nx, c->sm_count, cost);
    if ((rc = allow_max_smem(c, slice_fn(1, nae))) || (rc = allow_max_smem(c, slice_fn(2, nae)))) return rc;
  }
  const SliceGemm &w1 = s->g1[s->nvs - 1], &w2 = s->g2[s->nvs - 1];
  const size_t cols = (size_t)c->nk * c->na * s->nvs;
  if ((rc = salloc(c, &s->b1, w1.b_bytes())) || (rc = salloc(c, &s->b2, w2.b_bytes())) ||
      (rc = salloc(c, &s->m1, w1.b8_bytes())) || (rc = salloc(c, &s->m2, w2.b8_bytes())) ||
      (rc = salloc(c, &s->e1, cols)) || (rc = salloc(c, &s->e2, cols)) || (rc = salloc(c, &s->mx2, cols)) ||
      (rc = salloc(c, &s->ex2, (size_t)c->nx * c->na * s->nvs)) ||
      (rc = salloc(c, &s->d_err, 1)))
    return rc;
  OCN_CUDA(c, cudaMemsetAsync(s->d_err, 0, sizeof(int), c->stream));
  return OCN_OK;
}

int slice_splits(const ocn_ctx* c) { return c->slice ? c->slice->g2[0].p.ks : 1; }

// Vectors that one action's contractions take together.
int slice_width(const ocn_ctx* c) { return c->slice ? c->slice->nvs : 1; }

void slice_free(ocn_ctx* c) {
  SliceLR* s = c->slice;
  if (!s) return;
  slice_drop_a(c);
  slice_drop_mult(c);
  for (void* q : {(void*)s->b1, (void*)s->b2, (void*)s->m1, (void*)s->m2, (void*)s->e1, (void*)s->e2, (void*)s->mx2, (void*)s->ex2, (void*)s->d_err})
    if (q) cudaFree(q);
  delete s;
  c->slice = nullptr;
}

bool slice_ready(const ocn_ctx* c) { return c->slice && c->slice->ready; }

// Digit operands from d_u.  They take 3 bytes for every 2 of u, twice; when that
// is more than a quarter of the free device memory, or the caller declined them
// (ocn_set_fp64_digits), the context keeps the FP64-pipe kernels, which need only u.
int slice_set_bloch(ocn_ctx* c) {
  SliceLR* s = c->slice;
  if (!s) return OCN_OK;
  if (!(c->digits & 1) || (!s->g1[0].A && !slice_alloc_a(c, &s->g1[0], &s->g2[0], c->nx))) {
    slice_drop_a(c);
    return OCN_OK;
  }
  const size_t sx = (size_t)c->nk * c->nb, sk = c->nb;
  for (int sp = 0; sp < c->nspn; ++sp)
    if (int rc = slice_build(c, c->d_u + (size_t)sp * c->nx * sx, sx, sk, c->nx, s->g1[0], s->g2[0], sp)) return rc;
  OCN_CUDA(c, cudaStreamSynchronize(c->stream));
  s->ready = true;
  c->lr_xsplit = s->g2[0].p.ks;
  return OCN_OK;
}

// Digit operands of the projector coefficients c->mult.mpc [s][p][k*Nb + n]: the
// amplitudes are the band -> x contraction with the projectors in place of x, the
// back-projection the x -> band one with an operand shared by every k.  Grows the
// partial sums by the back-projection's slices.  Without the memory the context
// keeps the FP64-pipe multiplet kernels.  2p, 6^3 k / 64 bands / 128 projectors: the
// whole term 1200 us on the FP64 pipe (170 M complex multiply-adds) -> 80 us, a
// sixth of it the direct and exchange matrices (k_mult_hamp).
int slice_set_mult(ocn_ctx* c) {
  SliceLR* s = c->slice;
  if (!s) return OCN_OK;
  slice_drop_mult(c);
  const int np = c->mult.np;
  if (np == 0 || !(c->digits & 2)) return OCN_OK;
  slice_plan(&s->gm1, 1, c->na, c->na, c->nk, np, c->nb, c->sm_count, 0.0);
  slice_plan(&s->gm2, 2, c->na, c->na, c->nk, c->nb, np, c->sm_count, 32.0 * c->npsi / 6e12);
  s->gm2.p.bshared = 1;
  double* parts = nullptr;
  if (!slice_alloc_a(c, &s->gm1, &s->gm2, np) || salloc(c, &s->bm, s->gm2.b_bytes()) ||
      salloc(c, &s->mm, s->gm2.b8_bytes()) || salloc(c, &s->em, c->na) ||
      salloc(c, &s->mxm, c->na) || salloc(c, &s->amp_part, (size_t)c->nk * np * c->na) ||
      salloc(c, &parts, (size_t)(std::max(c->lr_xsplit_pipe, slice_splits(c)) + s->gm2.p.ks) * c->part_stride)) {
    slice_drop_mult(c);
    (void)cudaGetLastError();
    c->err.clear();
    return OCN_OK;
  }
  OCN_CUDA(c, cudaStreamSynchronize(c->stream));
  cudaFree(c->d_accpart);
  c->d_accpart = parts;
  c->mult_parts = s->gm2.p.ks;
  const size_t nbk = (size_t)c->nb * c->nk;
  for (int sp = 0; sp < c->nspn; ++sp)
    if (int rc = slice_build(c, c->mult.mpc + (size_t)sp * np * nbk, nbk, c->nb, np, s->gm1, s->gm2, sp)) return rc;
  OCN_CUDA(c, cudaStreamSynchronize(c->stream));
  s->mult_ready = true;
  return OCN_OK;
}

bool slice_mult_ready(const ocn_ctx* c) { return c->slice && c->slice->mult_ready; }

// psi operand of nv vectors (FP64 planes at stride vstride), shared by the amplitudes
// (nv = 1) and band -> x.
int slice_prep_psi(ocn_ctx* c, const double* d_pr, const double* d_pi, size_t vstride, int nv) {
  SliceLR* s = c->slice;
  const int nae = c->na * nv;
  TimedScope ts(c, T_LR_PREP);
  k_slice_prep_b1<<<c->nk, 256, 0, c->stream>>>(d_pr, d_pi, vstride, c->d_allow, c->nb, c->nk, c->na, nae, s->g1[0].p.Ge,
                                                slice_merged(nae) ? 1 : 0, s->b1, s->e1, s->mx2, s->m1, s->g1[0].s8());
  ++c->launches;
  OCN_CUDA(c, cudaGetLastError());
  return OCN_OK;
}

// The multiplet term of the one vector whose operand is in b1, into the d_accpart slices of vector v.
int slice_mult_apply(ocn_ctx* c, const double* d_pr, const double* d_pi, int v) {
  SliceLR* s = c->slice;
  MultDev& m = c->mult;
  TimedScope ts(c, T_MULT);
  int rc;
  const size_t nbk = (size_t)c->nb * c->nk;
  SliceColumns psi, hamp;
  psi.pr = d_pr;
  psi.pi = d_pi;
  hamp.f = m.hamp;
  if ((rc = slice_contract(c, s->gm1, s->gm1, s->b1, s->m1, s->e1, psi, m.mpc, m.np * nbk, nbk, c->nb, s->amp_part, nullptr)))
    return rc;
  const int n = m.np * c->na;
  k_slice_amp_reduce<<<(n + 31) / 32, 512, 0, c->stream>>>(s->amp_part, m.amp, c->nk, n);
  ++c->launches;
  OCN_CUDA(c, cudaGetLastError());
  if ((rc = mult_hamp(c, m.amp, m.hamp, 1))) return rc;
  k_slice_col_max<<<1, 512, 0, c->stream>>>(m.hamp, m.np, c->na, s->mxm);
  const int items = s->gm2.p.Ge * c->na * 4;
  k_slice_prep_b2<false><<<dim3((items + 255) / 256, 1), 256, 0, c->stream>>>(m.hamp, nullptr, m.np, c->na, s->gm2.p.Ge,
                                                                      slice_merged(c->na) ? 1 : 0, s->mxm, s->bm, s->em, s->mm, s->gm2.s8());
  c->launches += 2;
  OCN_CUDA(c, cudaGetLastError());
  double* part = c->d_accpart + (size_t)c->lr_xsplit * c->part_stride + (size_t)v * 2 * c->npsi;
  return slice_contract(c, s->gm2, s->gm2, s->bm, s->mm, s->em, hamp, m.mpc, m.np * nbk, nbk, c->nb, nullptr, part);
}

// phi[k][x][t] of the nv vectors whose operand is in b1, t = v*Na + a.
int slice_band_to_x(ocn_ctx* c, const double* d_pr, const double* d_pi, size_t vstride, double2* phi, int nv) {
  SliceLR* s = c->slice;
  TimedScope ts(c, T_LR_GEMM1);
  SliceColumns psi;
  psi.pr = d_pr;
  psi.pi = d_pi;
  psi.vstride = vstride;
  const size_t sx = (size_t)c->nk * c->nb;
  return slice_contract(c, s->g1[nv - 1], s->g1[0], s->b1, s->m1, s->e1, psi, c->d_u, c->nx * sx, sx, c->nb, phi, nullptr);
}

// Exponents per (x, t) and maxima per (k, t) that fx_transform leaves with phi' in
// integers; the maxima are cleared by slice_prep_psi.
void slice_exponents(ocn_ctx* c, int** ex, int** mx) {
  *ex = c->slice->ex2;
  *mx = c->slice->mx2;
}

// d_accpart slices of vectors v0 .. v0 + nv - 1 from phi'[k][x][t], in integers with
// slice_exponents or (not integers) in binary64.
int slice_x_to_band(ocn_ctx* c, const double2* phi, int nv, int v0, bool integers) {
  SliceLR* s = c->slice;
  const SliceGemm& g = s->g2[nv - 1];
  const int nae = c->na * nv;
  {
    TimedScope ts(c, T_LR_PREP);
    const int items = g.p.Ge * nae * 4, merged = slice_merged(nae) ? 1 : 0, s8 = g.s8();
    const dim3 grid((items + 255) / 256, c->nk);
    if (integers) {
      k_slice_prep_b2<true><<<grid, 256, 0, c->stream>>>(phi, s->ex2, c->nx, nae, g.p.Ge, merged, s->mx2, s->b2, s->e2, s->m2, s8);
    } else {
      k_slice_col_max<<<c->nk, 512, 0, c->stream>>>(phi, c->nx, nae, s->mx2);
      ++c->launches;
      k_slice_prep_b2<false><<<grid, 256, 0, c->stream>>>(phi, nullptr, c->nx, nae, g.p.Ge, merged, s->mx2, s->b2, s->e2, s->m2, s8);
    }
    ++c->launches;
    OCN_CUDA(c, cudaGetLastError());
  }
  TimedScope ts(c, T_LR_GEMM2);
  SliceColumns col;
  col.f = phi;
  col.ex = integers ? s->ex2 : nullptr;
  const size_t sx = (size_t)c->nk * c->nb;
  return slice_contract(c, g, s->g2[0], s->b2, s->m2, s->e2, col, c->d_u, c->nx * sx, sx, c->nb, nullptr,
                        c->d_accpart + (size_t)v0 * 2 * c->npsi);
}

int slice_set_starve(ocn_ctx* c, int on) {
  if (!c->slice) return set_err(c, OCN_ERR_STATE, "no FP64 tensor-core path");
  c->slice->starve = on ? 1 : 0;
  return OCN_OK;
}

const int* slice_err_word(const ocn_ctx* c) { return c->slice->d_err; }

// Reads and clears the device timeout flag (as mixed_check).
int slice_check(ocn_ctx* c) {
  if (!c->slice) return OCN_OK;
  int err = 0;
  OCN_CUDA(c, cudaMemcpyAsync(&err, c->slice->d_err, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  OCN_CUDA(c, cudaStreamSynchronize(c->stream));
  if (!err) return OCN_OK;
  OCN_CUDA(c, cudaMemset(c->slice->d_err, 0, sizeof(int)));
  return set_err(c, OCN_ERR_TIMEOUT, "tensor-core pipeline timed out (mask " + std::to_string(err) + ")");
}

}  // namespace ocn
