// ocn_fixed.cuh -- 64-bit block fixed point for the FP64 paths.
//
// GB300 issues 2 FP64 operations per clock and SM but 61 64-bit integer adds and
// 64 32x32->64 multiply-adds, so the arithmetic that has a common scale (digit
// slices of the contractions, the k-mesh transforms) runs on integers: values of
// one block share an exponent e (|v| < 2^e), an element is an integer multiple of
// 2^(e - F), and F is chosen so that at least 58 bits lie below the block's largest
// element -- more than the 53 of a binary64 value of that size.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

namespace ocn {

constexpr int FX_NAN = 0x40000000;  // block exponent of data that hold an Inf or NaN
constexpr int FX_BITS = 58;         // transform blocks: |int| < 2^58 before a pass (growth <= 8 sqrt 2 per pass)

// Magnitude bits of a value's high word: block maxima are taken over these.
__device__ __forceinline__ unsigned fx_mag(double v) { return (unsigned)__double2hiint(v) & 0x7fffffffu; }
// Block exponent e from the largest magnitude word: |v| < 2^e.
__device__ __forceinline__ int fx_exp(unsigned hw) {
  const int E = (int)(hw >> 20);
  return E == 0x7ff ? FX_NAN : E - 1022;
}
// v 2^(frac - e) rounded to nearest; 0 when e is FX_NAN.  |v| < 2^e, frac <= 62.
template <int FRAC>
__device__ __forceinline__ long long fx_from(double v, int e) {
  const long long b = __double_as_longlong(v);
  const int ev = (int)((b >> 52) & 0x7ff);
  unsigned long long m = (unsigned long long)b & 0xfffffffffffffull;
  if (ev) m |= 1ull << 52;
  const int s = max(ev, 1) - 1075 + FRAC - e;
  unsigned long long t = 0;
  if (s >= 0) t = m << min(s, FRAC - 53);  // s <= FRAC - 53 as |v| < 2^e
  else if (s > -54) t = (m + (1ull << (-s - 1))) >> (-s);
  if (e == FX_NAN) t = 0;
  return (long long)(b < 0 ? 0ull - t : t);
}
// Results outside the normal range (kept out of line: every caller is unrolled).
__device__ __noinline__ inline double fx_ldexp(long long v, int e) { return ldexp((double)v, e); }
// v 2^e rounded to binary64 (nearest even), |v| < 2^63: integer operations only --
// the hardware conversion runs on the FP64 pipe (it took 63 % of the transform).
__device__ __forceinline__ double fx_to_double(long long v, int e) {
  const unsigned long long u = (unsigned long long)(v < 0 ? -v : v);
  if (u == 0) return 0.0;
  const int lz = __clzll((long long)u);
  unsigned long long m = u << (lz - 1);        // top bit 62
  m += 0x1ffull + ((m >> 10) & 1ull);          // round to 53 bits
  m >>= 10;
  const int E = 1086 - lz + e;                 // biased exponent (the carry of the rounding adds to it)
  if (E >= 1 && E <= 2045) {
    const unsigned long long b = m + ((unsigned long long)(E - 1) << 52);
    return __longlong_as_double((long long)(b | ((unsigned long long)v & 0x8000000000000000ull)));
  }
  return fx_ldexp(v < 0 ? -(long long)m : (long long)m, e + 11 - lz);
}
// (h 2^30 + l) 2^e rounded to binary64; |h| < 2^56, |l| < 2^55
__device__ __forceinline__ double fx_to_double(long long h, long long l, int e) {
  h += l >> 30;
  unsigned ul = (unsigned)(l & 0x3fffffff);
  const bool neg = h < 0;
  if (neg) {  // magnitude: -(h 2^30 + l) = (-h - (l != 0)) 2^30 + (2^30 - l)
    h = -h - (ul ? 1 : 0);
    ul = (0x40000000u - ul) & 0x3fffffffu;
  }
  const unsigned top = (unsigned)((unsigned long long)h >> 34);       // above 64 bits
  const unsigned long long lo = ((unsigned long long)h << 30) | ul;
  const int s = top ? 33 - __clz((int)top) : (int)(lo >> 63);         // leaves at most 63 bits
  unsigned long long t = s ? ((unsigned long long)top << (64 - s)) | (lo >> s) : lo;
  if (lo & ((1ull << s) - 1ull)) t |= 1ull;                           // sticky: it only breaks ties
  const double r = fx_to_double((long long)t, e + s);
  return neg ? -r : r;
}

// c in (-1, 1) as q 2^-62 = h 2^-31 + l 2^-62
struct fxc {
  int h, l;
};
__host__ __device__ constexpr fxc fx_const(long long q) { return fxc{(int)(q >> 31), (int)(q & 0x7fffffff)}; }
// v c, |v| < 2^62, to about one unit
__device__ __forceinline__ long long fx_mul(long long v, int h, int l) {
  const int vh = (int)(v >> 31), vl = (int)(v & 0x7fffffff);
  const long long m = (long long)vh * l + (long long)vl * h;
  return (long long)vh * h + (m >> 31);
}
__device__ __forceinline__ long long fx_mul(long long v, fxc c) { return fx_mul(v, c.h, c.l); }

struct cfx {
  long long x, y;
};
__device__ __forceinline__ cfx operator+(cfx a, cfx b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ cfx operator-(cfx a, cfx b) { return {a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ cfx mul_i(cfx a) { return {-a.y, a.x}; }

// Backward DFT (exp(+2 pi i jm / N), unnormalised) of a line in registers; the
// forward one is the same on values with re and im exchanged.
template <int N>
__device__ __forceinline__ void fx_dft(cfx (&v)[N]) {
  if constexpr (N == 2) {
    const cfx a = v[0], b = v[1];
    v[0] = a + b;
    v[1] = a - b;
  } else if constexpr (N == 3) {
    constexpr fxc S = fx_const(3993837246235628775);  // sin 60
    const cfx t = v[1] + v[2], d = v[1] - v[2];
    const cfx m = {v[0].x - (t.x >> 1), v[0].y - (t.y >> 1)};
    const cfx s = mul_i(cfx{fx_mul(d.x, S), fx_mul(d.y, S)});
    v[0] = v[0] + t;
    v[1] = m + s;
    v[2] = m - s;
  } else if constexpr (N == 4) {
    const cfx s02 = v[0] + v[2], d02 = v[0] - v[2], s13 = v[1] + v[3], d13 = mul_i(v[1] - v[3]);
    v[0] = s02 + s13;
    v[2] = s02 - s13;
    v[1] = d02 + d13;
    v[3] = d02 - d13;
  } else if constexpr (N == 5) {
    constexpr fxc C1 = fx_const(1425089352415399811), C2 = fx_const(-3730932361629093763);  // cos 72, 144
    constexpr fxc S1 = fx_const(4385974038932618941), S2 = fx_const(2710681029835013083);   // sin 72, 144
    const cfx s1 = v[1] + v[4], d1 = v[1] - v[4], s2 = v[2] + v[3], d2 = v[2] - v[3];
    const cfx a1 = {v[0].x + fx_mul(s1.x, C1) + fx_mul(s2.x, C2), v[0].y + fx_mul(s1.y, C1) + fx_mul(s2.y, C2)};
    const cfx a2 = {v[0].x + fx_mul(s1.x, C2) + fx_mul(s2.x, C1), v[0].y + fx_mul(s1.y, C2) + fx_mul(s2.y, C1)};
    const cfx b1 = mul_i(cfx{fx_mul(d1.x, S1) + fx_mul(d2.x, S2), fx_mul(d1.y, S1) + fx_mul(d2.y, S2)});
    const cfx b2 = mul_i(cfx{fx_mul(d1.x, S2) - fx_mul(d2.x, S1), fx_mul(d1.y, S2) - fx_mul(d2.y, S1)});
    v[0] = v[0] + s1 + s2;
    v[1] = a1 + b1;
    v[4] = a1 - b1;
    v[2] = a2 + b2;
    v[3] = a2 - b2;
  } else if constexpr (N == 6) {  // prime factor 2 x 3: n = 3 n1 + 2 n2, k = 3 k1 + 4 k2 (mod 6)
    cfx p[3] = {v[0] + v[3], v[2] + v[5], v[4] + v[1]};
    cfx q[3] = {v[0] - v[3], v[2] - v[5], v[4] - v[1]};
    fx_dft<3>(p);
    fx_dft<3>(q);
    v[0] = p[0];
    v[4] = p[1];
    v[2] = p[2];
    v[3] = q[0];
    v[1] = q[1];
    v[5] = q[2];
  } else if constexpr (N == 7) {
    constexpr fxc C1 = fx_const(2875339201863983833), C2 = fx_const(-1026196679933739317),
                  C3 = fx_const(-4154985531143938469);  // cos 2 pi m / 7
    constexpr fxc S1 = fx_const(3605561316464170519), S2 = fx_const(4496061421583520199),
                  S3 = fx_const(2000935573311439104);   // sin 2 pi m / 7
    const cfx s1 = v[1] + v[6], s2 = v[2] + v[5], s3 = v[3] + v[4];
    const cfx d1 = v[1] - v[6], d2 = v[2] - v[5], d3 = v[3] - v[4];
    auto lin = [](cfx a, fxc ca, cfx b, fxc cb, cfx c, fxc cc) {
      return cfx{fx_mul(a.x, ca) + fx_mul(b.x, cb) + fx_mul(c.x, cc), fx_mul(a.y, ca) + fx_mul(b.y, cb) + fx_mul(c.y, cc)};
    };
    const cfx z{0, 0};
    const cfx a1 = v[0] + lin(s1, C1, s2, C2, s3, C3), a2 = v[0] + lin(s1, C2, s2, C3, s3, C1),
              a3 = v[0] + lin(s1, C3, s2, C1, s3, C2);
    const cfx b1 = mul_i(lin(d1, S1, d2, S2, d3, S3)), b2 = mul_i(lin(d1, S2, z - d2, S3, z - d3, S1)),
              b3 = mul_i(lin(d1, S3, z - d2, S1, d3, S2));
    v[0] = v[0] + s1 + s2 + s3;
    v[1] = a1 + b1;
    v[6] = a1 - b1;
    v[2] = a2 + b2;
    v[5] = a2 - b2;
    v[3] = a3 + b3;
    v[4] = a3 - b3;
  } else if constexpr (N == 8) {
    constexpr fxc H = fx_const(3260954456333195553);  // cos 45
    cfx e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    fx_dft<4>(e);
    fx_dft<4>(o);
    const cfx t1 = {fx_mul(o[1].x - o[1].y, H), fx_mul(o[1].y + o[1].x, H)};
    const cfx t2 = mul_i(o[2]);
    const cfx t3 = {-fx_mul(o[3].x + o[3].y, H), fx_mul(o[3].x - o[3].y, H)};
    v[0] = e[0] + o[0];
    v[4] = e[0] - o[0];
    v[1] = e[1] + t1;
    v[5] = e[1] - t1;
    v[2] = e[2] + t2;
    v[6] = e[2] - t2;
    v[3] = e[3] + t3;
    v[7] = e[3] - t3;
  } else {
    static_assert(N == 1, "line lengths 1..8");
  }
}

// Magnitude word of a pair (sign folded away): OR over a block bounds its largest element.
__device__ __forceinline__ unsigned fx_or(const cfx& a) {
  const int hx = (int)(a.x >> 32), hy = (int)(a.y >> 32);
  return (unsigned)(hx ^ (hx >> 31)) | (unsigned)(hy ^ (hy >> 31));
}
// Bits of the largest magnitude from the OR of the high words (an upper bound, 32 at least).
__device__ __forceinline__ int fx_nbits(unsigned orw) { return 64 - __clz((int)orw); }

// ---- passes of a block of transforms, four of them side by side (transform = lane mod 4)
// f(integral_constant of the line length): NC, or n (1..8) when NC is 0
template <int NC, class F>
__device__ __forceinline__ void fx_len(int n, F f) {
  if constexpr (NC > 0) {
    f(std::integral_constant<int, NC>{});
  } else {
    switch (n) {
      case 1: f(std::integral_constant<int, 1>{}); break;
      case 2: f(std::integral_constant<int, 2>{}); break;
      case 3: f(std::integral_constant<int, 3>{}); break;
      case 4: f(std::integral_constant<int, 4>{}); break;
      case 5: f(std::integral_constant<int, 5>{}); break;
      case 6: f(std::integral_constant<int, 6>{}); break;
      case 7: f(std::integral_constant<int, 7>{}); break;
      case 8: f(std::integral_constant<int, 8>{}); break;
    }
  }
}

template <int N>
__device__ __forceinline__ unsigned fx_or_line(const cfx (&v)[N]) {
  unsigned m = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) m |= fx_or(v[j]);
  return m;
}
// the four transforms' words of a pass: OR over the lanes of each class (lane mod 4)
__device__ __forceinline__ void fx_track(unsigned m, unsigned* word) {
  for (int o = 4; o < 32; o <<= 1) m |= __shfl_xor_sync(0xffffffffu, m, o);
  const int lane = threadIdx.x & 31;
  if (lane < 4) atomicOr(&word[lane], m);
}
// right shift that leaves 58 bits
__device__ __forceinline__ int fx_shift(unsigned orw) { return max(0, fx_nbits(orw) - FX_BITS); }

template <int N>
__device__ __forceinline__ void fx_load(cfx (&v)[N], const cfx* p, int st, int s) {
#pragma unroll
  for (int j = 0; j < N; ++j) {
    v[j] = p[j * st];
    v[j].x >>= s;
    v[j].y >>= s;
  }
}
template <int N>
__device__ __forceinline__ void fx_store(const cfx (&v)[N], cfx* p, int st) {
#pragma unroll
  for (int j = 0; j < N; ++j) p[j * st] = v[j];
}

}  // namespace ocn
