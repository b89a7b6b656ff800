// ocn_val_fx.cu -- the FP64 direct term of the valence action in 64-bit block
// fixed point (OCEAN_ladder.f90:155-1004; see ocn_valence.cu for the action):
//
//   T(y,k)   = sum_v A(x,v,k) conj(val(y,v,k))
//   T'(y,.)  = FFT_bwd[ ladder(.,x,y) o FFT_fwd[T(y,.)] ] / Nk
//   B(x,v,k) += sum_y T'(y,k) val(y,v,k)
//
// for k-meshes of 1..8 points per axis and up to 8 valence bands.  On the FP64 pipe
// (2 operations per clock and SM) the kernel is bound by it at any layout.  A, val, the ladder rows and each T have one
// scale, so products are formed from two 28/29-bit halves with 32x32->64 integer
// multiply-adds (high and middle partial sums; what is dropped is below 2^-58 of the
// largest product) and the transforms on integers (ocn_fixed.cuh, as
// ocn_fixfft.cu: shifted to 58 bits before every pass).  The sum over y is exact
// within a tile of four y and added in binary64 across tiles.
//
// Measured per action, 4 bands: 6^3 k / 7^3 x 9.37 -> 1.27 ms, 8^3 k / 10^3 x 84.7 ->
// 19.7 ms, 7x5x3 k / 210 x (3 bands, extents at run time) 1.96 -> 0.62 ms.  Bound by
// integer issue and the latency of the val rows from L2 (1.6 instructions per clock;
// 12 multiply-adds per complex product in T and again in B, about 700 instructions
// per k-point and pair).
//
// One CTA per x-point and y-range.  A tile of four y is processed by 4 lanes per
// line (t = lane mod 4 is the y): T is built on the k1 lines, transformed along
// k1, k2, k3, multiplied, transformed back, brought to one scale over the tile, and
// the B sums run with one thread per (k1 line, v), whose sums stay in registers.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "ocn_fixed.cuh"
#include "ocn_internal.h"

namespace ocn {

namespace {

constexpr int VF_FRAC = 57;  // A and val: |int| < 2^57 = 29-bit high and 28-bit low halves
constexpr int VF_LOW = 28;
constexpr int VF_HEAD = 2 * 8 * 4 * 4 + 64;  // shared words before A: two sets of pass maxima, block words
constexpr int VF_MAX_NV = 8;

__device__ __forceinline__ int4 vf_split(long long x, long long y) {
  constexpr long long mask = (1ll << VF_LOW) - 1;
  return make_int4((int)(x >> VF_LOW), (int)(x & mask), (int)(y >> VF_LOW), (int)(y & mask));
}
__device__ __forceinline__ void mad(long long& s, int a, int b) { s += (long long)a * b; }

// (h 2^28 + m) 2^e, |h|, |m| < 2^61: as many of the low bits as fit in 62 go along
__device__ __forceinline__ double vf_value(long long h, long long m, int e) {
  h += m >> VF_LOW;
  const int ml = (int)(m & ((1ll << VF_LOW) - 1));
  const int k = min(max(__clzll(h ^ (h >> 63)) - 2, 0), VF_LOW);
  return fx_to_double((long long)((unsigned long long)h << k) + (ml >> (VF_LOW - k)), e + VF_LOW - k);
}

struct VfParams {
  const double2* A;     // [x][v][k]
  const int4* V;        // [y][v][k] split halves (re high, low, im high, low)
  const int* eV;        // [y]
  const long long* L;   // [y][x][k]: ladder / Nk = L 2^(eL - 62)
  const int* eL;        // [y][x]
  double2* Bp;          // [ys][k][v][x]
  int nv, nx, yper;
  int n1, n2, n3;
};

// by 2^-s, s of either sign: mostly to the right, so the left shift is a warp-uniform detour
template <int N>
__device__ __forceinline__ void vf_scale(cfx (&v)[N], int s) {
  const int rs = min(max(s, 0), 63);
  if (__any_sync(__activemask(), s < 0)) {
    const int ls = max(-s, 0);
#pragma unroll
    for (int j = 0; j < N; ++j)
      v[j] = {(long long)((unsigned long long)v[j].x << ls), (long long)((unsigned long long)v[j].y << ls)};
  }
#pragma unroll
  for (int j = 0; j < N; ++j) v[j] = {v[j].x >> rs, v[j].y >> rs};
}

// Threads of a CTA and CTAs per SM the registers are held to, by cubic extent (0: any mesh).
constexpr int vf_cta(int n) { return n ? (4 * n * n + 31) / 32 * 32 : 256; }
constexpr int vf_min_ctas(int n) { return n == 0 ? 2 : (n == 8 ? 2 : (n == 6 ? 4 : (n == 5 ? 5 : 8))); }
// The B sums of a thread: in shared memory (fewer registers, more CTAs per SM), except 8^3,
// where two CTAs with them do not fit.
__host__ __device__ constexpr bool vf_acc_shared(int n) { return n != 8; }

// NV: valence bands known at compile time (0: from p), MAXC: (k1 line, v) pairs per thread
template <int N1, int N2, int N3, int NV, int MAXC>
__global__ void __launch_bounds__(vf_cta(N1), vf_min_ctas(N1)) k_val_ladder_fx(const VfParams p) {
  constexpr int NA = N1 ? N1 : 8;
  extern __shared__ __align__(16) unsigned char vfsm[];
  unsigned (*mxs)[8][4] = reinterpret_cast<unsigned (*)[8][4]>(vfsm);
  unsigned* blk = reinterpret_cast<unsigned*>(vfsm + 256);
  const int n1 = N1 ? N1 : p.n1, n2 = N2 ? N2 : p.n2, n3 = N3 ? N3 : p.n3;
  const int n23 = n2 * n3, nk = n1 * n23, nv = NV ? NV : p.nv;
  const int P3 = n3 | 1, slab = (n1 * n2 * P3 + 7) / 8 * 8 + 2;
  int4* As = reinterpret_cast<int4*>(vfsm + VF_HEAD);
  cfx* buf = reinterpret_cast<cfx*>(As + nv * nk);
  long long* Ls = reinterpret_cast<long long*>(buf + 4 * slab);  // ladder of the tile, [j][k3 line][y]
  const int x = blockIdx.x, ybeg = blockIdx.y * p.yper, yend = min(p.nx, ybeg + p.yper);
  const int t = threadIdx.x & 3, r = threadIdx.x >> 2;
  for (int i = threadIdx.x; i < 64; i += blockDim.x) reinterpret_cast<unsigned*>(vfsm)[i] = 0;
  if (threadIdx.x == 0) *blk = 0;
  __syncthreads();
  const double2* Ax = p.A + (size_t)x * nv * nk;
  {
    unsigned m = 0;
    for (int e = threadIdx.x; e < nv * nk; e += blockDim.x) m = max(m, max(fx_mag(Ax[e].x), fx_mag(Ax[e].y)));
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) atomicMax(blk, m);
  }
  __syncthreads();
  const int eA = fx_exp(*blk);
  for (int e = threadIdx.x; e < nv * nk; e += blockDim.x)
    As[e] = vf_split(fx_from<VF_FRAC>(Ax[e].x, eA), fx_from<VF_FRAC>(Ax[e].y, eA));

  cfx* bt = buf + t * slab;
  cfx* q1 = bt + (r / n3) * P3 + r % n3;
  cfx* q2 = bt + (r / n3) * n2 * P3 + r % n3;
  cfx* q3 = bt + r * P3;
  const bool on1 = r < n23, on2 = r < n1 * n3, on3 = r < n1 * n2;
  constexpr bool ACS = vf_acc_shared(N1);
  double2 acc[ACS ? 1 : MAXC][ACS ? 1 : NA];
  double2* accs = reinterpret_cast<double2*>(Ls + 4 * nk);  // [j][pair]
  const int npair = n23 * nv;
  if constexpr (ACS) {
    for (int i = threadIdx.x; i < npair * n1; i += blockDim.x) accs[i] = make_double2(0.0, 0.0);
  } else {
#pragma unroll
    for (int q = 0; q < MAXC; ++q)
#pragma unroll
      for (int j = 0; j < NA; ++j) acc[q][j] = make_double2(0.0, 0.0);
  }
  bool bad = eA == FX_NAN;
  __syncthreads();

  int par = 0;
  for (int y0 = ybeg; y0 < yend; y0 += 4, par ^= 1) {
    const int y = y0 + t;
    const bool ony = y < yend;
    const int yy = ony ? y : y0;  // padding lanes read a valid row and are left out
    const int eV = p.eV[yy], eL = p.eL[(size_t)yy * p.nx + x];
    unsigned (*mx)[4] = mxs[par];
    // the tile's ladder rows travel while T is built and transformed
    for (int i = threadIdx.x; i < 4 * nk; i += blockDim.x) {
      const int tl = i / nk, k = i - tl * nk, yl = min(y0 + tl, yend - 1);
      const unsigned dst = (unsigned)__cvta_generic_to_shared(Ls + ((k % n3) * (n1 * n2) + k / n3) * 4 + tl);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(p.L + ((size_t)yl * p.nx + x) * nk + k)
                   : "memory");
    }
    fx_len<N1>(n1, [&](auto ic) {  // T on the k1 lines, forward along k1 (re and im exchanged)
      constexpr int N = decltype(ic)::value;
      cfx v[N];
      unsigned m = 0;
      if (on1) {
        const int4* Vy = p.V + (size_t)yy * nv * nk + r;
        const int4* Ar = As + r;
#pragma unroll
        for (int j = 0; j < N; ++j) {
          long long hr = 0, mr = 0, hp = 0, mp = 0, hn = 0, mn = 0;  // re, im: positive and negative products
#pragma unroll
          for (int vv = 0; vv < (NV ? NV : VF_MAX_NV); ++vv) {
            if (NV == 0 && vv >= nv) break;
            const int4 b = __ldg(Vy + vv * nk + j * n23), a = Ar[vv * nk + j * n23];
            mad(hr, a.x, b.x);
            mad(hr, a.z, b.z);
            mad(mr, a.x, b.y);
            mad(mr, a.y, b.x);
            mad(mr, a.z, b.w);
            mad(mr, a.w, b.z);
            mad(hp, a.z, b.x);
            mad(hn, a.x, b.z);
            mad(mp, a.z, b.y);
            mad(mp, a.w, b.x);
            mad(mn, a.x, b.w);
            mad(mn, a.y, b.z);
          }
          v[j] = {hp - hn + ((mp - mn) >> VF_LOW), hr + (mr >> VF_LOW)};
        }
        m = fx_or_line<N>(v);
      }
      fx_track(m, mx[0]);
      __syncthreads();
      m = 0;
      if (on1) {
        vf_scale<N>(v, fx_shift(mx[0][t]));  // (bits below T's last do not exist)
        fx_dft<N>(v);
        fx_store<N>(v, q1, n2 * P3);
        m = fx_or_line<N>(v);
      }
      fx_track(m, mx[1]);
    });
    if (threadIdx.x < 32) mxs[par ^ 1][threadIdx.x >> 2][threadIdx.x & 3] = 0;  // the other set, last read a tile ago
    __syncthreads();
    fx_len<N2>(n2, [&](auto ic) {
      constexpr int N = decltype(ic)::value;
      unsigned m = 0;
      if (on2) {
        cfx v[N];
        fx_load<N>(v, q2, P3, fx_shift(mx[1][t]));
        fx_dft<N>(v);
        fx_store<N>(v, q2, P3);
        m = fx_or_line<N>(v);
      }
      fx_track(m, mx[2]);
    });
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    fx_len<N3>(n3, [&](auto ic) {  // forward along k3, ladder / Nk, backward along k3
      constexpr int N = decltype(ic)::value;
      cfx v[N];
      unsigned m = 0;
      if (on3) {
        const long long* w = Ls + 4 * r + t;
        fx_load<N>(v, q3, 1, fx_shift(mx[2][t]));
        fx_dft<N>(v);
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const long long wv = w[j * n1 * n2 * 4];
          const int wh = (int)(wv >> 31), wl = (int)(wv & 0x7fffffff);
          v[j] = {fx_mul(v[j].y, wh, wl), fx_mul(v[j].x, wh, wl)};
        }
        m = fx_or_line<N>(v);
      }
      fx_track(m, mx[3]);
      __syncthreads();
      m = 0;
      if (on3) {
        vf_scale<N>(v, fx_nbits(mx[3][t]) - FX_BITS);
        fx_dft<N>(v);
        fx_store<N>(v, q3, 1);
        m = fx_or_line<N>(v);
      }
      fx_track(m, mx[4]);
    });
    __syncthreads();
    fx_len<N2>(n2, [&](auto ic) {
      constexpr int N = decltype(ic)::value;
      unsigned m = 0;
      if (on2) {
        cfx v[N];
        fx_load<N>(v, q2, P3, fx_shift(mx[4][t]));
        fx_dft<N>(v);
        fx_store<N>(v, q2, P3);
        m = fx_or_line<N>(v);
      }
      fx_track(m, mx[5]);
    });
    __syncthreads();
    int etop;
    fx_len<N1>(n1, [&](auto ic) {  // backward along k1, then one scale for the four y
      constexpr int N = decltype(ic)::value;
      cfx v[N];
      unsigned m = 0;
      const int s5 = fx_shift(mx[5][t]);
      if (on1) {
        fx_load<N>(v, q1, n2 * P3, s5);
        fx_dft<N>(v);
        m = fx_or_line<N>(v);
      }
      fx_track(m, mx[6]);
      __syncthreads();
      // T' val = int 2^e (val int) 2^-57
      const int e = eA + 2 * eV + eL - 2 * VF_FRAC + 2 * VF_LOW + fx_shift(mx[0][t]) + fx_shift(mx[1][t]) +
                    fx_shift(mx[2][t]) + (fx_nbits(mx[3][t]) - FX_BITS) + fx_shift(mx[4][t]) + s5;
      const bool fin = eA != FX_NAN && eV != FX_NAN && eL != FX_NAN;
      etop = ony && fin ? e + fx_nbits(mx[6][t]) : -(1 << 28);
      etop = max(etop, __shfl_xor_sync(0xffffffffu, etop, 1));
      etop = max(etop, __shfl_xor_sync(0xffffffffu, etop, 2));
      if (__any_sync(0xffffffffu, ony && !fin)) bad = true;
      if (on1) {
        const bool use = ony && fin;
        vf_scale<N>(v, use ? etop - VF_FRAC - e : 0);  // |int| < 2^57
#pragma unroll
        for (int j = 0; j < N; ++j)
          *reinterpret_cast<int4*>(q1 + j * n2 * P3) = use ? vf_split(v[j].x, v[j].y) : make_int4(0, 0, 0, 0);
      }
    });
    __syncthreads();
    // B(x, v, k) += sum_y T'(y, k) val(y, v, k), exact over the tile
    const int ny = min(4, yend - y0);
#pragma unroll
    for (int q = 0; q < MAXC; ++q) {
      const int cb = threadIdx.x + q * blockDim.x;
      if (cb < npair) {
        const int vv = cb / n23, ln = cb - vv * n23;
        const int4* Tl = reinterpret_cast<const int4*>(buf + (ln / n3) * P3 + ln % n3);
        const int4* Vl = p.V + ((size_t)y0 * nv + vv) * nk + ln;
#pragma unroll
        for (int j = 0; j < NA; ++j) {
          if (N1 == 0 && j >= n1) continue;
          long long hp = 0, mp = 0, hn = 0, mn = 0, hi = 0, mi = 0;
#pragma unroll
          for (int yl = 0; yl < 4; ++yl) {  // T' of padding y is zero; its val row is read in range
            const int4 a = Tl[yl * slab + j * n2 * P3];
            const int4 b = __ldg(Vl + (size_t)min(yl, ny - 1) * nv * nk + j * n23);
            mad(hp, a.x, b.x);
            mad(hn, a.z, b.z);
            mad(mp, a.x, b.y);
            mad(mp, a.y, b.x);
            mad(mn, a.z, b.w);
            mad(mn, a.w, b.z);
            mad(hi, a.z, b.x);
            mad(hi, a.x, b.z);
            mad(mi, a.z, b.y);
            mad(mi, a.w, b.x);
            mad(mi, a.x, b.w);
            mad(mi, a.y, b.z);
          }
          const int eb = etop - 2 * VF_FRAC + VF_LOW;
          double2& d = ACS ? accs[j * npair + cb] : acc[ACS ? 0 : q][ACS ? 0 : j];
          d.x += vf_value(hp - hn, mp - mn, eb);
          d.y += vf_value(hi, mi, eb);
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < MAXC; ++q) {
    const int cb = threadIdx.x + q * blockDim.x;
    if (cb < n23 * nv) {
      const int vv = cb / n23, ln = cb - vv * n23;
#pragma unroll
      for (int j = 0; j < NA; ++j) {
        if (N1 == 0 && j >= n1) continue;
        double2 o = ACS ? accs[j * npair + cb] : acc[ACS ? 0 : q][ACS ? 0 : j];
        if (bad) o.x = o.y = __longlong_as_double(0x7ff8000000000000ll);
        p.Bp[(((size_t)blockIdx.y * nk + j * n23 + ln) * nv + vv) * p.nx + x] = o;
      }
    }
  }
}

// val [k][v][y] -> split halves [y][v][k] with one exponent per y (a CTA each)
__global__ void __launch_bounds__(256) k_vf_states(const double2* __restrict__ val, int nv, int nk, int nx,
                                                   int4* __restrict__ V, int* __restrict__ eV) {
  __shared__ unsigned sm;
  const int y = blockIdx.x;
  if (threadIdx.x == 0) sm = 0;
  __syncthreads();
  unsigned m = 0;
  for (int e = threadIdx.x; e < nv * nk; e += blockDim.x) {
    const double2 z = val[((size_t)(e % nk) * nv + e / nk) * nx + y];
    m = max(m, max(fx_mag(z.x), fx_mag(z.y)));
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(&sm, m);
  __syncthreads();
  const int ex = fx_exp(sm);
  for (int e = threadIdx.x; e < nv * nk; e += blockDim.x) {
    const double2 z = val[((size_t)(e % nk) * nv + e / nk) * nx + y];
    V[(size_t)y * nv * nk + e] = vf_split(fx_from<VF_FRAC>(z.x, ex), fx_from<VF_FRAC>(z.y, ex));
  }
  if (threadIdx.x == 0) eV[y] = ex;
}

// ladder rows (y, x) in place: binary64 -> ladder / Nk as 62-bit integers (a warp each)
__global__ void __launch_bounds__(256) k_vf_ladder(double* __restrict__ lad, size_t rows, int nk, int* __restrict__ eL) {
  const int lane = threadIdx.x & 31, a = 31 - __clz(nk);
  for (size_t w = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < rows; w += (size_t)gridDim.x * blockDim.x >> 5) {
    double* row = lad + w * nk;
    unsigned m = 0;
    for (int k = lane; k < nk; k += 32) m = max(m, fx_mag(row[k]));
    m = __reduce_max_sync(0xffffffffu, m);
    const int e = fx_exp(m);
    for (int k = lane; k < nk; k += 32) {
      const long long q = fx_from<62>(row[k], e);
      reinterpret_cast<long long*>(row)[k] = (long long)(((__int128)q << a) / nk);
    }
    if (lane == 0) eL[w] = e == FX_NAN ? FX_NAN : e - a;
  }
}

typedef void (*VfFn)(const VfParams);
template <int NV, int MAXC>
VfFn vf_fn(const int n[3]) {
  if (n[0] == n[1] && n[1] == n[2]) switch (n[0]) {
      case 3: return k_val_ladder_fx<3, 3, 3, NV, MAXC>;
      case 4: return k_val_ladder_fx<4, 4, 4, NV, MAXC>;
      case 5: return k_val_ladder_fx<5, 5, 5, NV, MAXC>;
      case 6: return k_val_ladder_fx<6, 6, 6, NV, MAXC>;
      case 8: return k_val_ladder_fx<8, 8, 8, NV, MAXC>;
    }
  return k_val_ladder_fx<0, 0, 0, NV, MAXC>;
}

int vf_threads(const int n[3]) {
  const int lines = std::max({n[1] * n[2], n[0] * n[2], n[0] * n[1]});
  return (4 * lines + 31) / 32 * 32;
}
// four bands (one pair per thread) unrolled; other counts at run time
VfFn vf_select(const int n[3], int nv) {
  if (nv == 4) return vf_fn<4, 1>(n);
  return n[1] * n[2] * nv <= vf_threads(n) ? vf_fn<0, 1>(n) : vf_fn<0, 2>(n);
}

size_t vf_smem(const int n[3], int nv) {
  const int slab = (n[0] * n[1] * (n[2] | 1) + 7) / 8 * 8 + 2;
  const size_t nk = (size_t)n[0] * n[1] * n[2];
  const bool cube8 = n[0] == 8 && n[1] == 8 && n[2] == 8;
  return VF_HEAD + (nv * nk + 4 * (size_t)slab) * 16 + 4 * nk * 8 + (cube8 ? 0 : nv * nk * 16);
}

}  // namespace

bool val_fx_supported(const int kmesh[3], int nv, size_t smem_optin) {
  for (int i = 0; i < 3; ++i)
    if (kmesh[i] > 8) return false;
  return nv <= VF_MAX_NV && kmesh[1] * kmesh[2] * nv <= 2 * vf_threads(kmesh) && vf_smem(kmesh, nv) <= smem_optin;
}

// Raises the kernel's shared-memory limit; CTAs per SM.
cudaError_t val_fx_plan(const int kmesh[3], int nv, size_t smem_optin, int* per_sm) {
  VfFn f = vf_select(kmesh, nv);
  cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_optin);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, f, vf_threads(kmesh), vf_smem(kmesh, nv));
}

void val_fx_states(const double2* val, int nv, int nk, int nx, void* V, int* eV, cudaStream_t s) {
  k_vf_states<<<nx, 256, 0, s>>>(val, nv, nk, nx, static_cast<int4*>(V), eV);
}
void val_fx_ladder(double* lad, size_t rows, int nk, int* eL, int sm_count, cudaStream_t s) {
  k_vf_ladder<<<(unsigned)std::min<size_t>((rows + 7) / 8, (size_t)16 * sm_count), 256, 0, s>>>(lad, rows, nk, eL);
}
void val_fx_apply(const int kmesh[3], int nv, int nx, int yper, int ysplit, const double2* A, const void* V,
                  const int* eV, const void* lad, const int* eL, double2* Bp, cudaStream_t s) {
  const VfParams p = {A, static_cast<const int4*>(V), eV, static_cast<const long long*>(lad), eL, Bp, nv, nx, yper,
                      kmesh[0], kmesh[1], kmesh[2]};
  vf_select(kmesh, nv)<<<dim3(nx, ysplit), vf_threads(kmesh), vf_smem(kmesh, nv), s>>>(p);
}

}  // namespace ocn
