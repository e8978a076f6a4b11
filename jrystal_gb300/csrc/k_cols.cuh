// Column kernels (see fft_cols.cuh): x transforms of the sphere's (y, z) columns,
// one instantiation per length and precision.
#pragma once
#include <algorithm>

#include "fft_cols.cuh"

namespace jrg {
namespace cols {

// kinetic table |G+k|^2/2 in the path's precision (FP32: the plan's FP32 copy)
template <typename R> using TK_t = std::conditional_t<sizeof(R) == 4, float, double>;
template <typename R> const TK_t<R>* tk_table(const jrg_plan* P) {
  if constexpr (sizeof(R) == 4) return P->d.tkf;
  else return P->d.tk;
}

constexpr int kColThreads = 64;

// ---- sphere -> T: x inverse of every column -----------------------------------
// need: bands of weight zero are left out (their columns are not read later)
template <typename R, int NX>
__global__ void __launch_bounds__(kColThreads, (sizeof(R) == 4 && NX <= 64) ? 6 : 1) k_cols_inv(
    const C_t<R>* __restrict__ coef, C_t<R>* __restrict__ T, const int* __restrict__ xmap,
    const double* __restrict__ need, int ncol, int tp, int ng, int nbands, int bpt) {
  using C = C_t<R>;
  constexpr int H = win_half<NX>();
  const int col = blockIdx.x * kColThreads + threadIdx.x;
  if (col >= ncol) return;
  const int b_end = min(nbands, (int)(blockIdx.y + 1) * bpt);
#pragma unroll 1
  for (int b = blockIdx.y * bpt; b < b_end; ++b) {
    if (need[b] == 0.0) continue;
    const C* cb = coef + (size_t)b * ng;
    C* out = T + (size_t)b * NX * tp + col;
    line_fft<C, NX, +1, H>(
        [&](auto ii) {
          const int e = xmap[win_pos<NX, H>(ii.value) * ncol + col];
          return e >= 0 ? cb[e] : czero<C>();
        },
        [&](auto kk, C v) { out[(size_t)kk.value * tp] = v; });
  }
}

// ---- T -> g_C: x forward, kinetic term, weights --------------------------------
//   g[b][e] = w_b (tk[k][e] c[b][e] + scale FFT(V psi_b)[e])
// Each thread copies the coefficients and kinetic values of its column to its
// own places in shared memory while the column's T values are in flight, so
// that a line waits for memory once (64^3, 648 bands: 135 us with the reads next
// to the stores).
template <typename R, int NX>
__global__ void __launch_bounds__(kColThreads) k_cols_fwd(
    const C_t<R>* __restrict__ T, const C_t<R>* __restrict__ coef, C_t<R>* __restrict__ gcoef,
    const double* __restrict__ wband, const TK_t<R>* __restrict__ tk, const int* __restrict__ xmap, int ncol,
    int tp, int nb_per_k, int band0, int ng, int nk, double scale, int nbands, int bpt) {
  using C = C_t<R>;
  using TK = TK_t<R>;
  constexpr int H = win_half<NX>(), W = win_n<NX>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* sc = reinterpret_cast<C*>(smem_raw) + threadIdx.x;             // [W][threads]
  TK* st = reinterpret_cast<TK*>(smem_raw + sizeof(C) * W * kColThreads) + threadIdx.x;
  int* se = reinterpret_cast<int*>(smem_raw + (sizeof(C) + sizeof(TK)) * W * kColThreads) + threadIdx.x;
  const int col = blockIdx.x * kColThreads + threadIdx.x;
  if (col >= ncol) return;
  const int b_begin = blockIdx.y * bpt, b_end = min(nbands, b_begin + bpt);
  double wd = wband[band0 + b_begin];
#pragma unroll
  for (int j = 0; j < W; ++j) se[j * kColThreads] = xmap[j * ncol + col];
  const R scl = (R)scale;
#pragma unroll 1
  for (int b = b_begin; b < b_end; ++b) {
    const int gb = band0 + b;
    const double wb = wd;
    if (b + 1 < b_end) wd = wband[gb + 1];
    C* g_out = gcoef + (size_t)b * ng;
    if (wb == 0.0) {   // an empty band has no gradient
#pragma unroll 8
      for (int j = 0; j < W; ++j) {
        const int e = se[j * kColThreads];
        if (e >= 0) g_out[e] = czero<C>();
      }
      continue;
    }
    const R w = (R)wb;
    const TK* tkk = tk + (size_t)((gb / nb_per_k) % nk) * ng;
    const C* cb = coef + (size_t)b * ng;
#pragma unroll
    for (int j = 0; j < W; ++j) {
      const int e = max(se[j * kColThreads], 0);
      cp_async<sizeof(C)>(sc + j * kColThreads, cb + e);
      cp_async<sizeof(TK)>(st + j * kColThreads, tkk + e);
    }
    cp_async_commit();
    const C* in = T + (size_t)b * NX * tp + col;
    C v[W];
    line_fft<C, NX, -1, -1>([&](auto ii) { return in[(size_t)ii.value * tp]; },
                            [&](auto kk, C q) {
                              if constexpr (in_win<NX, H>(kk.value)) v[win_pos<NX, H>(kk.value)] = q;
                            });
    cp_async_wait<0>();
#pragma unroll
    for (int j = 0; j < W; ++j) {
      const int e = se[j * kColThreads];
      const C c = sc[j * kColThreads];
      const R t = (R)st[j * kColThreads];
      C g;
      g.x = w * (t * c.x + scl * v[j].x);
      g.y = w * (t * c.y + scl * v[j].y);
      if (e >= 0) g_out[e] = g;
    }
  }
}

// bands per thread: a few while the grid still fills the GPU several times over
inline int bands_per_thread(int blocks, int nbands) {
  int bpt = 4;
  while (bpt > 1 && (long long)blocks * nbands < 152LL * 12 * bpt) bpt /= 2;
  return bpt;
}

template <typename R, int N> int run_columns(const jrg_plan* P, int op, const fast::Args& a, cudaStream_t st) {
  using C = C_t<R>;
  const int cb = (P->ncol + kColThreads - 1) / kColThreads;
  const int bpt = bands_per_thread(cb, a.nbands);
  const dim3 grid(cb, (a.nbands + bpt - 1) / bpt);
  if (op == fast::OP_PLANE_INV) {
    k_cols_inv<R, N><<<grid, kColThreads, 0, st>>>(reinterpret_cast<const C*>(a.in), reinterpret_cast<C*>(a.out),
                                                   P->d.xmap, a.w, P->ncol, P->tpitch, P->ng, a.nbands, bpt);
    return launched("k_cols_inv");
  }
  const size_t sm = (sizeof(C) + sizeof(TK_t<R>) + sizeof(int)) * (size_t)win_n<N>() * kColThreads;
  int rc;
  if ((rc = prep((const void*)k_cols_fwd<R, N>, sm)) <= 0) return rc;
  k_cols_fwd<R, N><<<grid, kColThreads, sm, st>>>(
      reinterpret_cast<const C*>(a.in), reinterpret_cast<const C*>(a.aux), reinterpret_cast<C*>(a.out), a.w,
      tk_table<R>(P), P->d.xmap, P->ncol, P->tpitch, P->nb, a.band0, P->ng, P->nk, a.wscale, a.nbands, bpt);
  return launched("k_cols_fwd");
}

}  // namespace cols
}  // namespace jrg
