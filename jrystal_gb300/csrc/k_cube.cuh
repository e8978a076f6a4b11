// Slab kernels of cubic grids N^3 (see fft_cols.cuh): the phases of
// cols_lines.cuh inlined, with the pitch known at compile time and the density
// sums in registers.  At 64^3 (Si8, 27 k-points, 432 occupied bands) the density
// pass takes 139 us and the adjoint pass 258 us, against 283 and 433 us with the
// phases as functions: calls save and restore the registers that a line fills.
#pragma once
#include "cols_lines.cuh"

namespace jrg {
namespace cols {

// 168 registers hold an FP32 line of 64 of the adjoint pass, or half a line of 96
// of either pass (density at 96^3: 2.32 ms with 256 threads, 1.46 with 384), or an
// FP64 line of 32 (energy and gradient of 48 bands, 256 threads and 384: 25^3 634 and
// 611 us, 27^3 628 and 603, 30^3 708 and 681)
template <typename R, int N> __host__ __device__ constexpr int cube_apply_threads() {
  return sizeof(R) == 4 || N <= 32 ? 384 : 256;
}
// the z phase of the adjoint pass by pairs of threads (FP64, bound by its
// arithmetic, gains nothing: 48^3 414 us, by pairs 440)
template <typename R, int N> __host__ __device__ constexpr bool cube_pairs() {
  return sizeof(R) == 4 && halves<R, N>();
}
template <typename R, int N> __host__ __device__ constexpr int cube_density_threads() {
  return sizeof(R) == 4 && N > 64 ? 384 : 256;
}

template <typename R, int N>
__global__ void __launch_bounds__(cube_density_threads<R, N>())
k_cube_density(C_t<R>* __restrict__ T, R* __restrict__ rho_part, const double* __restrict__ wband, double wscale,
               int band0, int nband, int bands_per_group, const short* __restrict__ col_of, int tp, int tile, int sub,
               double* __restrict__ gscale, const int* __restrict__ bad, int nbad) {
  using C = C_t<R>;
  constexpr int H = win_half<N>(), W = win_n<N>(), parts = halves<R, N>() ? 2 : 1, M = N / parts, PV = N | 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const SlabLayout<R> lay(tile, N, N, 0, bands_per_group, true, false);
  R* sum = reinterpret_cast<R*>(smem_raw + lay.grid);
  R* sw = reinterpret_cast<R*>(smem_raw + lay.w);
  short* scol = reinterpret_cast<short*>(smem_raw + lay.col);
  unsigned short* list = reinterpret_cast<unsigned short*>(smem_raw + lay.list);
  __shared__ int count;
  const int x = blockIdx.x, grp = blockIdx.y, tid = threadIdx.x;
  const int b_begin = grp * bands_per_group, b_end = min(nband, b_begin + bands_per_group);
  live_bands(wband + band0, b_begin, b_end, list, &count);
  group_weights<R>(wband + band0, b_begin, b_end, wscale, gscale, grp, sw, bad + (size_t)grp * nbad, nbad);
  for (int i = tid; i < W * W; i += blockDim.x) scol[i] = col_of[i];
  __syncthreads();
  const int nl = count;
  Tile<C> q;
  q.bstride = (size_t)N * tp;
  q.src = T + (size_t)b_begin * q.bstride + (size_t)x * tp;
  q.m = 0;
  q.col = (int)lay.col;
  q.wz = W;
  q.pz = W;
  const int s = tid / (parts * N), yp = tid - s * (parts * N);
  const int par = yp / N, y = yp - par * N;
  R acc[M];
#pragma unroll
  for (int k = 0; k < M; ++k) acc[k] = (R)0;
#pragma unroll 1
  for (int b0 = 0; b0 < nl; b0 += tile) {
    q.n = min(tile, nl - b0);
    q.list = (int)lay.list + b0 * (int)sizeof(unsigned short);
    y_inverse_body<C, N, W>(q);
    __syncthreads();
    prefetch_tile<C>(q.src, list + b0 + tile, min(tile, nl - b0 - tile), tp, q.bstride);
    if (s < sub) {
#pragma unroll 1
      for (int t = s; t < q.n; t += sub) {
        const C* row = reinterpret_cast<const C*>(smem_raw) + (t * N + y) * W;
        const R w = sw[list[b0 + t]];
        auto load = [&](auto ii) { return row[win_pos<N, H>(ii.value)]; };
        auto store = [&](auto kk, C v) { acc[kk.value] += w * (v.x * v.x + v.y * v.y); };
        if constexpr (parts == 2) ln::half_inverse<C, N, H>(par, load, store);
        else line_fft<C, N, +1, H>(load, store);
      }
    }
    __syncthreads();
  }
#pragma unroll 1
  for (int p = 0; p < sub; ++p) {
    if (s == p) {
      R* d = sum + y * PV + par;
#pragma unroll
      for (int k = 0; k < M; ++k) d[parts * k] = p == 0 ? acc[k] : d[parts * k] + acc[k];
    }
    __syncthreads();
  }
  R* out = rho_part + ((size_t)grp * N + x) * (N * N);
  for (int i = tid; i < N * N; i += blockDim.x) {
    const int yy = i / N;
    out[i] = sum[yy * PV + i - yy * N];
  }
}

template <typename R, int N>
__global__ void __launch_bounds__(cube_apply_threads<R, N>())
k_cube_apply_v(C_t<R>* __restrict__ T, const R* __restrict__ vr, const double* __restrict__ need, int nband,
               int bands_per_group, const short* __restrict__ col_of, int ncol, int tp, int tile, int sub) {
  using C = C_t<R>;
  constexpr int W = win_n<N>(), PV = N | 1;
  constexpr bool places = halves<R, N>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const SlabLayout<R> lay(tile, N, N, ncol, bands_per_group, false, places);
  R* sv = reinterpret_cast<R*>(smem_raw + lay.grid);
  int* spos = reinterpret_cast<int*>(smem_raw + lay.pos);   // place of a column's y forward output
  short* scol = reinterpret_cast<short*>(smem_raw + lay.col);
  unsigned short* list = reinterpret_cast<unsigned short*>(smem_raw + lay.list);
  __shared__ int count;
  const int x = blockIdx.x, grp = blockIdx.y, tid = threadIdx.x;
  const int b_begin = grp * bands_per_group, b_end = min(nband, b_begin + bands_per_group);
  live_bands(need, b_begin, b_end, list, &count);
  column_places<places>(col_of, scol, spos, N, W, W, W);
  for (int i = tid; i < N * N; i += blockDim.x) {
    const int y = i / N;
    sv[y * PV + i - y * N] = vr[(size_t)x * (N * N) + i];
  }
  __syncthreads();
  const int nl = count;
  Tile<C> q;
  q.bstride = (size_t)N * tp;
  q.src = T + (size_t)b_begin * q.bstride + (size_t)x * tp;
  q.m = 0;
  q.col = (int)lay.col;
  q.wz = W;
  q.pz = W;
#pragma unroll 1
  for (int b0 = 0; b0 < nl; b0 += tile) {
    q.n = min(tile, nl - b0);
    q.list = (int)lay.list + b0 * (int)sizeof(unsigned short);
    y_inverse_body<C, N, W>(q);
    __syncthreads();
    prefetch_tile<C>(q.src, list + b0 + tile, min(tile, nl - b0 - tile), tp, q.bstride);
    if constexpr (cube_pairs<R, N>()) z_apply_pairs<C, N, W>(q, (int)lay.grid, PV, sub);
    else z_apply_body<C, N, W>(q, (int)lay.grid, N, PV, sub);
    __syncthreads();
    y_forward_body<C, N, W>(q);
    __syncthreads();
    if constexpr (places) {
      columns_back<C>(q, list + b0, spos, ncol, N, W);
      __syncthreads();
    }
  }
}

template <typename R, int N> int run_cube(const jrg_plan* P, int op, const fast::Args& a, cudaStream_t st) {
  if constexpr (!cube_used<R, N>()) {
    return 0;
  } else {
    using C = C_t<R>;
    const int bpg = a.bands_per_group, groups = (a.nbands + bpg - 1) / bpg;
    constexpr int ylines = (halves<R, N>() ? 2 : 1) * win_n<N>();
    int rc;
    if (op == fast::OP_LINE_DENSITY) {
      const SlabShape s = slab_shape((halves<R, N>() ? 2 : 1) * N, ylines, std::min(a.nbands, bpg), cube_density_threads<R, N>(),
                                     [&](int tile) { return SlabLayout<R>(tile, N, N, 0, bpg, true, false).total; });
      if ((rc = prep((const void*)k_cube_density<R, N>, s.smem)) <= 0) return rc;
      k_cube_density<R, N><<<dim3(N, groups), s.threads, s.smem, st>>>(
          reinterpret_cast<C*>(const_cast<void*>(a.in)), reinterpret_cast<R*>(a.out), a.w, a.wscale, a.band0, a.nbands,
          bpg, P->d.col_of, P->tpitch, s.tile, s.sub, a.gscale, a.bad, a.nbad);
      return launched("k_cube_density");
    }
    const SlabShape s = slab_shape((cube_pairs<R, N>() ? 2 : 1) * N, ylines, std::min(a.nbands, bpg), cube_apply_threads<R, N>(), [&](int tile) {
      return SlabLayout<R>(tile, N, N, P->ncol, bpg, false, halves<R, N>()).total;
    });
    if ((rc = prep((const void*)k_cube_apply_v<R, N>, s.smem)) <= 0) return rc;
    k_cube_apply_v<R, N><<<dim3(N, groups), s.threads, s.smem, st>>>(
        reinterpret_cast<C*>(a.out), reinterpret_cast<const R*>(a.aux), a.w, a.nbands, bpg, P->d.col_of, P->ncol,
        P->tpitch, s.tile, s.sub);
    return launched("k_cube_apply_v");
  }
}

}  // namespace cols
}  // namespace jrg
