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

// ---- T -> g_C: x forward, kinetic term, weights (odd lengths) ------------------
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

// Even lengths, two threads a column: each transforms the even or the
// odd x of the column (fft_line.cuh, half lines), they exchange through shared
// memory what the other needs, and the even one writes the outputs k <= H, the odd
// one k >= NX - H.  Half the registers a thread, so that more warps wait for memory
// at a time: Si8 64^3 115 -> 102 us, Si8 48^3 16 -> 12, Si2 48^3 FP64 59 -> 41.  CTAs
// on an SM: 64^3 three 102 us, four 107; 48^3 three 14, four 12.
template <typename R, int NX>
__global__ void __launch_bounds__(2 * kColThreads, sizeof(R) == 8 ? 2 : (NX <= 48 ? 4 : 3)) k_cols_fwd_pair(
    const C_t<R>* __restrict__ T, const C_t<R>* __restrict__ coef, C_t<R>* __restrict__ gcoef,
    const double* __restrict__ wband, const TK_t<R>* __restrict__ tk, const int* __restrict__ xmap, int ncol,
    int tp, int nb_per_k, int band0, int ng, int nk, double scale, int nbands, int bpt) {
  using C = C_t<R>;
  using TK = TK_t<R>;
  constexpr int H = win_half<NX>(), M = NX / 2, HO = H + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int c64 = threadIdx.x % kColThreads, par = threadIdx.x / kColThreads;
  C* ex = reinterpret_cast<C*>(smem_raw) + c64;   // [2 H + 1][columns]: O'[0 .. H], then E[M - H .. M - 1]
  const int col = blockIdx.x * kColThreads + c64;
  const bool act = col < ncol;
  const int mine = par ? H : HO, pos0 = par ? HO : 0;   // this thread's window positions
  const int b_begin = blockIdx.y * bpt, b_end = min(nbands, b_begin + bpt);
  double wd = wband[band0 + b_begin];
  int e[HO];
#pragma unroll
  for (int j = 0; j < HO; ++j) e[j] = act && j < mine ? xmap[(pos0 + j) * ncol + col] : -1;
  const R scl = (R)scale;
#pragma unroll 1
  for (int b = b_begin; b < b_end; ++b) {
    const int gb = band0 + b;
    const double wb = wd;
    if (b + 1 < b_end) wd = wband[gb + 1];
    C* g_out = gcoef + (size_t)b * ng;
    if (wb == 0.0) {   // an empty band has no gradient
#pragma unroll
      for (int j = 0; j < HO; ++j)
        if (e[j] >= 0) g_out[e[j]] = czero<C>();
      continue;
    }
    const R w = (R)wb;
    const TK* tkk = tk + (size_t)((gb / nb_per_k) % nk) * ng;
    const C* cb = coef + (size_t)b * ng;
    const C* in = T + ((size_t)b * NX + par) * tp + (act ? col : 0);
    C o[M];
    ln::half_forward<C, NX>(par, [&](auto ii) { return in[(size_t)(2 * ii.value) * tp]; },
                            [&](auto kk, C v) { o[kk.value] = v; });
    __syncthreads();   // the last band's exchange has been read
    if (par) {
#pragma unroll
      for (int j = 0; j < HO; ++j) ex[j * kColThreads] = o[j];
    } else {
#pragma unroll
      for (int j = 0; j < H; ++j) ex[(HO + j) * kColThreads] = o[M - H + j];
    }
    __syncthreads();
    C x[HO];
    if (par) {
#pragma unroll
      for (int j = 0; j < H; ++j) x[j] = ln::vsub(ex[(HO + j) * kColThreads], o[M - H + j]);
      x[H] = czero<C>();
    } else {
#pragma unroll
      for (int j = 0; j < HO; ++j) x[j] = ln::vadd(o[j], ex[j * kColThreads]);
    }
    C c[HO];
    R t[HO];
#pragma unroll
    for (int j = 0; j < HO; ++j) {
      c[j] = cb[max(e[j], 0)];
      t[j] = (R)tkk[max(e[j], 0)];
    }
#pragma unroll
    for (int j = 0; j < HO; ++j) {
      C g;
      g.x = w * (t[j] * c[j].x + scl * x[j].x);
      g.y = w * (t[j] * c[j].y + scl * x[j].y);
      if (e[j] >= 0) g_out[e[j]] = g;
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
  int rc;
  if constexpr (N % 2 == 0) {
    const size_t smx = sizeof(C) * (size_t)win_n<N>() * kColThreads;
    if ((rc = prep((const void*)k_cols_fwd_pair<R, N>, smx)) <= 0) return rc;
    k_cols_fwd_pair<R, N><<<grid, 2 * kColThreads, smx, st>>>(
        reinterpret_cast<const C*>(a.in), reinterpret_cast<const C*>(a.aux), reinterpret_cast<C*>(a.out), a.w,
        tk_table<R>(P), P->d.xmap, P->ncol, P->tpitch, P->nb, a.band0, P->ng, P->nk, a.wscale, a.nbands, bpt);
    return launched("k_cols_fwd_pair");
  } else {
    const size_t sm = (sizeof(C) + sizeof(TK_t<R>) + sizeof(int)) * (size_t)win_n<N>() * kColThreads;
    if ((rc = prep((const void*)k_cols_fwd<R, N>, sm)) <= 0) return rc;
    k_cols_fwd<R, N><<<grid, kColThreads, sm, st>>>(
        reinterpret_cast<const C*>(a.in), reinterpret_cast<const C*>(a.aux), reinterpret_cast<C*>(a.out), a.w,
        tk_table<R>(P), P->d.xmap, P->ncol, P->tpitch, P->nb, a.band0, P->ng, P->nk, a.wscale, a.nbands, bpt);
    return launched("k_cols_fwd");
  }
}

}  // namespace cols
}  // namespace jrg
