// ocn_val_fx.cu -- the FP64 direct term of the valence action (OCEAN_ladder.f90:155-1004;
// see ocn_valence.cu for the action):
//
//   T(y,k)   = sum_v A(x,v,k) conj(val(y,v,k))
//   T'(y,.)  = FFT_bwd[ ladder(.,x,y) o FFT_fwd[T(y,.)] ] / Nk
//   B(x,v,k) += sum_y T'(y,k) val(y,v,k)
//
// for k-meshes of 1..8 points per axis and up to 8 valence bands, with the products in
// binary64 and the transforms on 64-bit integers (block fixed point, ocn_fixed.cuh, as
// ocn_fixfft.cu: shifted to 58 bits before every pass).  GB300 issues 2 FP64 operations per
// clock and SM; a transform mixes the elements of a block, so its error is relative to the
// block's largest element in any arithmetic and 58 bits hold more than binary64, while the
// products are not: with the products on integers as well, A and val at 57 bits of the
// largest element of a point, the sums lost accuracy wherever the two were graded
// oppositely over the bands or T' and val over y.
//
// Measured per action, 4 bands: 6^3 k / 7^3 x 9.37 ms with everything on the FP64 pipe, 1.86 ms
// now (1.27 with the products on integers); 8^3 k / 10^3 x 84.7, 32.0 (19.7); 7x5x3 k / 210 x
// (3 bands, extents at run time) 1.96, 0.75 (0.62).  Bound by the FP64 pipe: the 32 multiply-adds
// per k-point and pair take 1.39 of the 1.86 ms; the transforms' integers run beside them.
//
// One CTA per x-point and y-range.  A tile of four y is processed by 4 lanes per
// line (t = lane mod 4 is the y): T is built on the k1 lines, transformed along
// k1, k2, k3, multiplied, transformed back, and the B sums run with one thread per
// (k1 line, v).
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "ocn_fixed.cuh"
#include "ocn_internal.h"

namespace ocn {

namespace {

constexpr int VF_HEAD = 2 * 8 * 4 * 4;  // shared words before A: two sets of pass maxima
constexpr int VF_MAX_NV = 8;

struct VfParams {
  const double2* A;     // [x][v][k]
  const double2* V;     // [y][v][k]
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
  const int n1 = N1 ? N1 : p.n1, n2 = N2 ? N2 : p.n2, n3 = N3 ? N3 : p.n3;
  const int n23 = n2 * n3, nk = n1 * n23, nv = NV ? NV : p.nv;
  const int P3 = n3 | 1, slab = (n1 * n2 * P3 + 7) / 8 * 8 + 2;
  double2* As = reinterpret_cast<double2*>(vfsm + VF_HEAD);
  cfx* buf = reinterpret_cast<cfx*>(As + nv * nk);
  long long* Ls = reinterpret_cast<long long*>(buf + 4 * slab);  // ladder of the tile, [j][k3 line][y]
  const int x = blockIdx.x, ybeg = blockIdx.y * p.yper, yend = min(p.nx, ybeg + p.yper);
  const int t = threadIdx.x & 3, r = threadIdx.x >> 2;
  for (int i = threadIdx.x; i < 64; i += blockDim.x) reinterpret_cast<unsigned*>(vfsm)[i] = 0;
  const double2* Ax = p.A + (size_t)x * nv * nk;
  for (int e = threadIdx.x; e < nv * nk; e += blockDim.x) As[e] = Ax[e];

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
  __syncthreads();

  int par = 0;
  for (int y0 = ybeg; y0 < yend; y0 += 4, par ^= 1) {
    const int y = y0 + t;
    const bool ony = y < yend;
    const int yy = ony ? y : y0;  // padding lanes read a valid row and are left out
    const int eL = p.eL[(size_t)yy * p.nx + x];
    int e0 = 0;  // |T| < 2^e0
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
      double2 T[N];
      unsigned m = 0;
      if (on1) {
        const double2* Vy = p.V + (size_t)yy * nv * nk + r;
        const double2* Ar = As + r;
#pragma unroll
        for (int j = 0; j < N; ++j) {
          double re = 0.0, im = 0.0;
#pragma unroll
          for (int vv = 0; vv < (NV ? NV : VF_MAX_NV); ++vv) {
            if (NV == 0 && vv >= nv) break;
            const double2 b = __ldg(Vy + vv * nk + j * n23), a = Ar[vv * nk + j * n23];
            re = __fma_rn(a.x, b.x, re);
            im = __fma_rn(a.y, b.x, im);
            re = __fma_rn(a.y, b.y, re);
            im = __fma_rn(-a.x, b.y, im);
          }
          T[j] = make_double2(re, im);
          m = max(m, max(fx_mag(re), fx_mag(im)));
        }
      }
      for (int o = 4; o < 32; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
      if ((threadIdx.x & 31) < 4) atomicMax(&mx[0][threadIdx.x & 3], m);
      __syncthreads();
      e0 = fx_exp(mx[0][t]);
      m = 0;
      if (on1) {
        cfx v[N];
#pragma unroll
        for (int j = 0; j < N; ++j) v[j] = {fx_from<FX_BITS>(T[j].y, e0), fx_from<FX_BITS>(T[j].x, e0)};
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
    fx_len<N1>(n1, [&](auto ic) {  // backward along k1, to binary64
      constexpr int N = decltype(ic)::value;
      if (!on1) return;
      cfx v[N];
      const int s5 = fx_shift(mx[5][t]);
      fx_load<N>(v, q1, n2 * P3, s5);
      fx_dft<N>(v);
      const int e = e0 - FX_BITS + eL + fx_shift(mx[1][t]) + fx_shift(mx[2][t]) + (fx_nbits(mx[3][t]) - FX_BITS) +
                    fx_shift(mx[4][t]) + s5;
      const bool fin = e0 != FX_NAN && eL != FX_NAN;
#pragma unroll
      for (int j = 0; j < N; ++j) {
        double2 z = make_double2(fx_to_double(v[j].x, e), fx_to_double(v[j].y, e));
        if (!fin) z.x = z.y = __longlong_as_double(0x7ff8000000000000ll);
        *reinterpret_cast<double2*>(q1 + j * n2 * P3) = z;
      }
    });
    __syncthreads();
    // B(x, v, k) += sum_y T'(y, k) val(y, v, k)
    const int ny = min(4, yend - y0);
#pragma unroll
    for (int q = 0; q < MAXC; ++q) {
      const int cb = threadIdx.x + q * blockDim.x;
      if (cb < npair) {
        const int vv = cb / n23, ln = cb - vv * n23;
        const double2* Tl = reinterpret_cast<const double2*>(buf + (ln / n3) * P3 + ln % n3);
        const double2* Vl = p.V + ((size_t)y0 * nv + vv) * nk + ln;
#pragma unroll
        for (int j = 0; j < NA; ++j) {
          if (N1 == 0 && j >= n1) continue;
          double2& d = ACS ? accs[j * npair + cb] : acc[ACS ? 0 : q][ACS ? 0 : j];
          double2 s = d;
#pragma unroll
          for (int yl = 0; yl < 4; ++yl) {
            if (yl >= ny) break;
            const double2 a = Tl[yl * slab + j * n2 * P3];
            const double2 b = __ldg(Vl + (size_t)yl * nv * nk + j * n23);
            s.x = __fma_rn(a.x, b.x, s.x);
            s.y = __fma_rn(a.y, b.x, s.y);
            s.x = __fma_rn(-a.y, b.y, s.x);
            s.y = __fma_rn(a.x, b.y, s.y);
          }
          d = s;
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
        const double2 o = ACS ? accs[j * npair + cb] : acc[ACS ? 0 : q][ACS ? 0 : j];
        p.Bp[(((size_t)blockIdx.y * nk + j * n23 + ln) * nv + vv) * p.nx + x] = o;
      }
    }
  }
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
// Four bands (one pair per thread) unrolled; other counts at run time: the FP64 pipe bounds
// both (6^3 k / 7^3 x: 1.29, 1.61, 3.19 ms with 2, 3, 6 bands, 1.86 with 4).
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

void val_fx_ladder(double* lad, size_t rows, int nk, int* eL, int sm_count, cudaStream_t s) {
  k_vf_ladder<<<(unsigned)std::min<size_t>((rows + 7) / 8, (size_t)16 * sm_count), 256, 0, s>>>(lad, rows, nk, eL);
}
void val_fx_apply(const int kmesh[3], int nv, int nx, int yper, int ysplit, const double2* A, const double2* V,
                  const void* lad, const int* eL, double2* Bp, cudaStream_t s) {
  const VfParams p = {A, V, static_cast<const long long*>(lad), eL, Bp, nv, nx, yper, kmesh[0], kmesh[1], kmesh[2]};
  vf_select(kmesh, nv)<<<dim3(nx, ysplit), vf_threads(kmesh), vf_smem(kmesh, nv), s>>>(p);
}

}  // namespace ocn
