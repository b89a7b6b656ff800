// ocn_fixfft.cu -- the FP64 k-mesh transform of the long-range term in 64-bit
// block fixed point:
//
//   phi'(.,x,t) = FFT_fwd[ W(.,x) o FFT_bwd[ phi(.,x,t) ] ] / Nk
//
// (long_range.f90:928-939, FFTW signs, Modules/FFT_wrapper.f90:24-25) for k-meshes
// of 1..8 points per axis.  In binary64 the transform is bound by the FP64 pipe (2
// operations per clock and SM: 319 us for the 6912 transforms of 8^3 points of the
// 8^3 k / 12^3 x 1s case, 766 us for 12000 of 6^3).  All values of one transform
// have one scale, so the butterflies are integer adds and the few real products
// 62-bit constants (ocn_fixed.cuh).  Before every pass the block is shifted so that
// its largest element takes 58 bits -- the pass may grow it by 8 sqrt 2 -- which
// keeps at least five bits more than binary64 has below the largest element; the
// rounding error is smaller than that of the binary64 transform, which rounds to
// 53 bits at every butterfly.
//
// One CTA per x-point and four transforms, one thread per (line, transform) of a
// pass: k1, k2, k3 backward, W, k3, k2, k1 forward.  The outer k1 passes read and
// write HBM from registers, the others exchange lines through shared memory (16
// bytes per complex value, odd line pitch and slabs of 2 mod 8 units: no bank
// conflicts).  W / Nk is kept as 62-bit integers with one exponent per x-point, so
// the normalisation costs nothing.  The pass maxima that set the shifts are
// OR-reductions over the four lanes' classes (t = lane mod 4) and four shared words.
// For the digit contractions the result stays integers, with one exponent per (x, t)
// and the exponent maxima per (k, t) that scale the next operand collected on the way
// out: rounding to binary64 and back took an eighth of the instructions.
//
// Measured: 319 -> 60 us (8^3, 6912 transforms), 766 -> 53 us (6^3, 12000), 375 ->
// 32 us (7x6x5, 3960 of the 11880 of three vectors).  Bound by integer issue (about 3000
// instructions per thread), not by the 114 MB it moves.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "ocn_fixed.cuh"
#include "ocn_internal.h"

namespace ocn {

namespace {

constexpr int FX_HEAD = 96;     // shared memory before the lines: six passes x four words

struct FxParams {
  double2* phi;                 // [k][x][t], transformed in place
  const long long* W;           // [x][k]: W / Nk = W 2^(we - 62)
  const int* we;                // [x]
  int* ex;                      // integer output: phi' = int 2^ex[x][t], ...
  int* mx;                      // ... and running maxima over x of the exponents e, |phi'(k,x,t)| <= 2^e, [k][t]
  int nx, ld;
  int n1, n2, n3;
};

// N1, N2, N3: mesh extents known at compile time (0: from p).  INT: phi' stays integers
// (re, im as 64-bit words in phi's place) for the digit operand of the next contraction.
template <int N1, int N2, int N3, bool INT>
__global__ void __launch_bounds__(256, 3) k_fx_transform(const FxParams p) {
  extern __shared__ __align__(16) unsigned char fxsm[];
  unsigned (*mx)[4] = reinterpret_cast<unsigned (*)[4]>(fxsm);  // [pass][transform]
  cfx* buf = reinterpret_cast<cfx*>(fxsm + FX_HEAD);
  const int n1 = N1 ? N1 : p.n1, n2 = N2 ? N2 : p.n2, n3 = N3 ? N3 : p.n3;
  const int P3 = n3 | 1;
  const int slab = (n1 * n2 * P3 + 7) / 8 * 8 + 2;
  const int x = blockIdx.x, t = threadIdx.x & 3, r = threadIdx.x >> 2;
  const int tg = blockIdx.y * 4 + t;
  if (threadIdx.x < 24) mx[threadIdx.x >> 2][threadIdx.x & 3] = 0;
  __syncthreads();
  cfx* bt = buf + t * slab;
  const int n23 = n2 * n3;
  // line r of each pass: k1 lines (k2, k3), k2 lines (k1, k3), k3 lines (k1, k2)
  cfx* q1 = bt + (r / n3) * P3 + r % n3;
  cfx* q2 = bt + (r / n3) * n2 * P3 + r % n3;
  cfx* q3 = bt + r * P3;
  const bool on1 = r < n23, on2 = r < n1 * n3, on3 = r < n1 * n2;
  int e0 = 0;

  fx_len<N1>(n1, [&](auto ic) {  // k1 backward, from HBM
    constexpr int N = decltype(ic)::value;
    double2 in[N];
    unsigned m = 0;
    if (on1) {
#pragma unroll
      for (int j = 0; j < N; ++j) in[j] = p.phi[((size_t)(j * n23 + r) * p.nx + x) * p.ld + tg];
#pragma unroll
      for (int j = 0; j < N; ++j) m = max(m, max(fx_mag(in[j].x), fx_mag(in[j].y)));
    }
    for (int o = 4; o < 32; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) < 4) atomicMax(&mx[0][threadIdx.x & 3], m);
    __syncthreads();
    e0 = fx_exp(mx[0][t]);
    m = 0;
    if (on1) {
      cfx v[N];
#pragma unroll
      for (int j = 0; j < N; ++j) v[j] = {fx_from<FX_BITS>(in[j].x, e0), fx_from<FX_BITS>(in[j].y, e0)};
      fx_dft<N>(v);
      fx_store<N>(v, q1, n2 * P3);
      m = fx_or_line<N>(v);
    }
    fx_track(m, mx[1]);
  });
  __syncthreads();
  fx_len<N2>(n2, [&](auto ic) {  // k2 backward
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
  __syncthreads();
  int s3 = 0;
  fx_len<N3>(n3, [&](auto ic) {  // k3 backward, W / Nk, k3 forward (re and im exchanged from here on)
    constexpr int N = decltype(ic)::value;
    cfx v[N];
    unsigned m = 0;
    if (on3) {
      const long long* w = p.W + (size_t)x * n1 * n23 + r * n3;
      fx_load<N>(v, q3, 1, fx_shift(mx[2][t]));
      fx_dft<N>(v);
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const long long wv = __ldg(w + j);
        const int wh = (int)(wv >> 31), wl = (int)(wv & 0x7fffffff);
        v[j] = {fx_mul(v[j].y, wh, wl), fx_mul(v[j].x, wh, wl)};
      }
      m = fx_or_line<N>(v);
    }
    fx_track(m, mx[3]);
    __syncthreads();
    s3 = fx_nbits(mx[3][t]) - FX_BITS;
    m = 0;
    if (on3) {
      const int rs = max(s3, 0), ls = max(-s3, 0);
#pragma unroll
      for (int j = 0; j < N; ++j) v[j] = {(long long)((unsigned long long)v[j].x << ls) >> rs, (long long)((unsigned long long)v[j].y << ls) >> rs};
      fx_dft<N>(v);
      fx_store<N>(v, q3, 1);
      m = fx_or_line<N>(v);
    }
    fx_track(m, mx[4]);
  });
  __syncthreads();
  fx_len<N2>(n2, [&](auto ic) {  // k2 forward
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
  fx_len<N1>(n1, [&](auto ic) {  // k1 forward, to HBM
    constexpr int N = decltype(ic)::value;
    if (!on1) return;
    cfx v[N];
    const int s5 = fx_shift(mx[5][t]), we = p.we[x];
    fx_load<N>(v, q1, n2 * P3, s5);
    fx_dft<N>(v);
    const bool bad = e0 == FX_NAN || we == FX_NAN;
    const int e = e0 - FX_BITS + we + fx_shift(mx[1][t]) + fx_shift(mx[2][t]) + s3 + fx_shift(mx[4][t]) + s5;
    if (INT && r == 0) p.ex[(size_t)x * p.ld + tg] = bad ? FX_NAN : e;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const int k = j * n23 + r;
      const size_t o = ((size_t)k * p.nx + x) * p.ld + tg;
      if constexpr (INT) {
        reinterpret_cast<longlong2*>(p.phi)[o] = make_longlong2(v[j].y, v[j].x);
        const unsigned long long m = (unsigned long long)((v[j].x ^ (v[j].x >> 63)) | (v[j].y ^ (v[j].y >> 63)));
        const int em = bad ? FX_NAN : e + 64 - __clzll((long long)m);
        int* d = p.mx + (size_t)k * p.ld + tg;  // the running maximum rarely grows: look before the atomic
        if (em > __ldcg(d)) atomicMax(d, em);
      } else {
        double2 z = make_double2(fx_to_double(v[j].y, e), fx_to_double(v[j].x, e));
        if (bad) z.x = z.y = __longlong_as_double(0x7ff8000000000000ll);
        p.phi[o] = z;
      }
    }
  });
}

typedef void (*FxFn)(const FxParams);
template <bool INT>
FxFn fx_fn(const int n[3]) {
  if (n[0] == n[1] && n[1] == n[2]) switch (n[0]) {
      case 2: return k_fx_transform<2, 2, 2, INT>;
      case 3: return k_fx_transform<3, 3, 3, INT>;
      case 4: return k_fx_transform<4, 4, 4, INT>;
      case 5: return k_fx_transform<5, 5, 5, INT>;
      case 6: return k_fx_transform<6, 6, 6, INT>;
      case 7: return k_fx_transform<7, 7, 7, INT>;
      case 8: return k_fx_transform<8, 8, 8, INT>;
    }
  return k_fx_transform<0, 0, 0, INT>;
}

// W / Nk as 62-bit integers, one exponent per x-point (a CTA each).
__global__ void __launch_bounds__(128) k_fx_w(const double* __restrict__ W, int nk, long long* __restrict__ out,
                                              int* __restrict__ we) {
  __shared__ unsigned sm;
  const int x = blockIdx.x;
  if (threadIdx.x == 0) sm = 0;
  __syncthreads();
  unsigned m = 0;
  for (int k = threadIdx.x; k < nk; k += blockDim.x) m = max(m, fx_mag(W[(size_t)x * nk + k]));
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(&sm, m);
  __syncthreads();
  const int e = fx_exp(sm), a = 31 - __clz(nk);  // 2^a <= Nk
  for (int k = threadIdx.x; k < nk; k += blockDim.x) {
    const long long q = fx_from<62>(W[(size_t)x * nk + k], e);
    out[(size_t)x * nk + k] = (long long)(((__int128)q << a) / nk);
  }
  if (threadIdx.x == 0) we[x] = e == FX_NAN ? FX_NAN : e - a;
}

size_t fx_smem(const int n[3]) {
  const int slab = (n[0] * n[1] * (n[2] | 1) + 7) / 8 * 8 + 2;
  return FX_HEAD + (size_t)4 * slab * sizeof(cfx);
}

}  // namespace

// Extents 1..8 per axis: lines fit in registers and one thread per line in a CTA.
bool fx_supported(const ocn_ctx* c) {
  for (int i = 0; i < 3; ++i)
    if (c->dims.kmesh[i] > 8) return false;
  return c->d_Wfx != nullptr && c->na % 4 == 0;
}

int fx_init(ocn_ctx* c) {
  for (int i = 0; i < 3; ++i)
    if (c->dims.kmesh[i] > 8) return OCN_OK;
  cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&c->d_Wfx), (size_t)c->nk * c->nx * sizeof(long long));
  if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&c->d_Wexp), (size_t)c->nx * sizeof(int));
  if (e != cudaSuccess) return set_err(c, OCN_ERR_ALLOC, std::string("cudaMalloc: ") + cudaGetErrorString(e));
  if (int rc = allow_max_smem(c, fx_fn<true>(c->dims.kmesh))) return rc;
  return allow_max_smem(c, fx_fn<false>(c->dims.kmesh));
}

int fx_set_w(ocn_ctx* c) {
  if (!c->d_Wfx) return OCN_OK;
  k_fx_w<<<c->nx, 128, 0, c->stream>>>(c->d_W, c->nk, c->d_Wfx, c->d_Wexp);
  ++c->launches;
  OCN_CUDA(c, cudaGetLastError());
  OCN_CUDA(c, cudaStreamSynchronize(c->stream));
  return OCN_OK;
}

// phi[k][x][t], t < nt, in place.  ex, mx null: binary64; else integers with exponents
// ex[x][t] and column maxima mx[k][t] (cleared by the caller).
int fx_transform(ocn_ctx* c, double2* phi, int nt, int* ex, int* mx) {
  const int* n = c->dims.kmesh;
  const FxParams p = {phi, c->d_Wfx, c->d_Wexp, ex, mx, c->nx, nt, n[0], n[1], n[2]};
  const int lines = std::max({n[1] * n[2], n[0] * n[2], n[0] * n[1]});
  (ex ? fx_fn<true>(n) : fx_fn<false>(n))<<<dim3(c->nx, nt / 4), (4 * lines + 31) / 32 * 32, fx_smem(n), c->stream>>>(p);
  ++c->launches;
  OCN_CUDA(c, cudaGetLastError());
  return OCN_OK;
}

}  // namespace ocn
