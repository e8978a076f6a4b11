// Slab kernels and dispatch of the column-first transforms (fft_cols.cuh).
#include "fft_cols.cuh"

namespace jrg {
namespace cols {

// ---- density pass over the x slabs ---------------------------------------------
template <typename R>
__global__ void __launch_bounds__(kDensityThreads)
k_slab_density(C_t<R>* __restrict__ T, R* __restrict__ rho_part, const double* __restrict__ wband, double wscale,
               int band0, int nband, int bands_per_group, const short* __restrict__ col_of, int ny, int nz, int tp,
               int tile, int sub, double* __restrict__ gscale, const int* __restrict__ bad, int nbad) {
  using C = C_t<R>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const SlabLayout<R> lay(tile, ny, nz, 0, bands_per_group, true, false);
  R* sum = reinterpret_cast<R*>(smem_raw + lay.grid);
  R* sw = reinterpret_cast<R*>(smem_raw + lay.w);
  short* scol = reinterpret_cast<short*>(smem_raw + lay.col);
  unsigned short* list = reinterpret_cast<unsigned short*>(smem_raw + lay.list);
  __shared__ int count;
  const int x = blockIdx.x, nx = gridDim.x, grp = blockIdx.y, tid = threadIdx.x;
  const int b_begin = grp * bands_per_group, b_end = min(nband, b_begin + bands_per_group);
  live_bands(wband + band0, b_begin, b_end, list, &count);
  group_weights<R>(wband + band0, b_begin, b_end, wscale, gscale, grp, sw, bad + (size_t)grp * nbad, nbad);
  for (int i = tid; i < window(ny) * window(nz); i += blockDim.x) scol[i] = col_of[i];
  for (int i = tid; i < ny * lay.pv; i += blockDim.x) sum[i] = (R)0;
  __syncthreads();
  const int nl = count;
  Tile<C> q;
  q.bstride = (size_t)nx * tp;
  q.src = T + (size_t)b_begin * q.bstride + (size_t)x * tp;
  q.m = 0;
  q.col = (int)lay.col;
  q.wz = window(nz);
  q.pz = lay.pz;
#pragma unroll 1
  for (int b0 = 0; b0 < nl; b0 += tile) {
    q.n = min(tile, nl - b0);
    q.list = (int)lay.list + b0 * (int)sizeof(unsigned short);
    switch (ny) {
#define CASE(N) case N: y_inverse<C, N>(q); break;
      JRG_COLS_SIZES(CASE)
#undef CASE
    }
    __syncthreads();
    prefetch_tile<C>(q.src, list + b0 + tile, min(tile, nl - b0 - tile), tp, q.bstride);
    switch (nz) {
#define CASE(N) case N: z_density<C, N>(q, (int)lay.w, (int)lay.grid, ny, lay.pv, sub); break;
      JRG_COLS_SIZES(CASE)
#undef CASE
    }
    __syncthreads();
  }
  R* out = rho_part + ((size_t)grp * nx + x) * ((size_t)ny * nz);
  for (int i = tid; i < ny * nz; i += blockDim.x) {
    const int y = i / nz;
    out[i] = sum[y * lay.pv + i - y * nz];
  }
}

template <typename R> int launch_density(const jrg_plan* P, const fast::Args& a, cudaStream_t st) {
  using C = C_t<R>;
  const SlabShape s = slab_shape(parts_of<R>(P->nz) * P->ny, parts_of<R>(P->ny) * window(P->nz),
                                 std::min(a.nbands, a.bands_per_group), kDensityThreads, [&](int tile) {
                                   return SlabLayout<R>(tile, P->ny, P->nz, 0, a.bands_per_group, true, false).total;
                                 });
  int rc;
  if ((rc = prep((const void*)k_slab_density<R>, s.smem)) <= 0) return rc;
  const int groups = (a.nbands + a.bands_per_group - 1) / a.bands_per_group;
  k_slab_density<R><<<dim3(P->nx, groups), s.threads, s.smem, st>>>(
      reinterpret_cast<C*>(const_cast<void*>(a.in)), reinterpret_cast<R*>(a.out), a.w, a.wscale, a.band0, a.nbands,
      a.bands_per_group, P->d.col_of, P->ny, P->nz, P->tpitch, s.tile, s.sub, a.gscale, a.bad, a.nbad);
  return launched("k_slab_density");
}

// ---- adjoint pass over the x slabs ---------------------------------------------
template <typename R>
__global__ void __launch_bounds__(kApplyThreads)
k_slab_apply_v(C_t<R>* __restrict__ T, const R* __restrict__ vr, const double* __restrict__ need, int nband,
               int bands_per_group, const short* __restrict__ col_of, int ny, int nz, int ncol, int tp, int tile,
               int sub) {
  using C = C_t<R>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const bool places = parts_of<R>(ny) == 2;
  const SlabLayout<R> lay(tile, ny, nz, ncol, bands_per_group, false, places);
  R* sv = reinterpret_cast<R*>(smem_raw + lay.grid);
  int* spos = reinterpret_cast<int*>(smem_raw + lay.pos);   // place of a column's y forward output
  short* scol = reinterpret_cast<short*>(smem_raw + lay.col);
  unsigned short* list = reinterpret_cast<unsigned short*>(smem_raw + lay.list);
  __shared__ int count;
  const int x = blockIdx.x, nx = gridDim.x, grp = blockIdx.y, tid = threadIdx.x;
  const int b_begin = grp * bands_per_group, b_end = min(nband, b_begin + bands_per_group);
  const int wy = window(ny), wz = window(nz);
  live_bands(need, b_begin, b_end, list, &count);
  if (places) column_places<true>(col_of, scol, spos, ny, wy, wz, lay.pz);
  else column_places<false>(col_of, scol, spos, ny, wy, wz, lay.pz);
  for (int i = tid; i < ny * nz; i += blockDim.x) {
    const int y = i / nz;
    sv[y * lay.pv + i - y * nz] = vr[(size_t)x * ny * nz + i];
  }
  __syncthreads();
  const int nl = count;
  Tile<C> q;
  q.bstride = (size_t)nx * tp;
  q.src = T + (size_t)b_begin * q.bstride + (size_t)x * tp;
  q.m = 0;
  q.col = (int)lay.col;
  q.wz = wz;
  q.pz = lay.pz;
#pragma unroll 1
  for (int b0 = 0; b0 < nl; b0 += tile) {
    q.n = min(tile, nl - b0);
    q.list = (int)lay.list + b0 * (int)sizeof(unsigned short);
    switch (ny) {
#define CASE(N) case N: y_inverse<C, N>(q); break;
      JRG_COLS_SIZES(CASE)
#undef CASE
    }
    __syncthreads();
    prefetch_tile<C>(q.src, list + b0 + tile, min(tile, nl - b0 - tile), tp, q.bstride);
    switch (nz) {
#define CASE(N) case N: z_apply<C, N>(q, (int)lay.grid, ny, lay.pv, sub); break;
      JRG_COLS_SIZES(CASE)
#undef CASE
    }
    __syncthreads();
    switch (ny) {
#define CASE(N) case N: y_forward<C, N>(q); break;
      JRG_COLS_SIZES(CASE)
#undef CASE
    }
    __syncthreads();
    if (places) {
      columns_back<C>(q, list + b0, spos, ncol, ny, lay.pz);
      __syncthreads();
    }
  }
}

template <typename R> int launch_apply(const jrg_plan* P, const fast::Args& a, cudaStream_t st) {
  using C = C_t<R>;
  const int bpg = a.bands_per_group;
  const SlabShape s = slab_shape(P->ny, parts_of<R>(P->ny) * window(P->nz), std::min(a.nbands, bpg), kApplyThreads,
                                 [&](int tile) {
                                   return SlabLayout<R>(tile, P->ny, P->nz, P->ncol, bpg, false,
                                                        parts_of<R>(P->ny) == 2).total;
                                 });
  int rc;
  if ((rc = prep((const void*)k_slab_apply_v<R>, s.smem)) <= 0) return rc;
  const int groups = (a.nbands + bpg - 1) / bpg;
  k_slab_apply_v<R><<<dim3(P->nx, groups), s.threads, s.smem, st>>>(
      reinterpret_cast<C*>(a.out), reinterpret_cast<const R*>(a.aux), a.w, a.nbands, bpg, P->d.col_of, P->ny, P->nz,
      P->ncol, P->tpitch, s.tile, s.sub);
  return launched("k_slab_apply_v");
}

// ---- dispatch -------------------------------------------------------------------
static bool length_ok(int n) {
  switch (n) {
#define CASE(N) case N: return true;
    JRG_COLS_SIZES(CASE)
#undef CASE
    default: return false;
  }
}

bool covers(int prec, int nx, int ny, int nz, int nb, bool inside, bool pruned) {
  // FP64 is bound by its arithmetic, and here the adjoint pass repeats the y
  // inverse: the plane-first kernels keep the cubic sizes whose known zeros they
  // leave out (32^3, 243 bands of an Al cell: 974 us for the four passes, 1085 us
  // column-first; 48^3, not pruned there: 1237 and 762 us)
  if (prec == 64 && pruned) return false;
  if (!inside || !length_ok(nx) || !length_ok(ny) || !length_ok(nz)) return false;
  // one band of either slab kernel has to fit the shared memory
  if (nb > 65535) return false;
  const int ncol = window(ny) * window(nz);
  const size_t least = prec == 64 ? SlabLayout<double>(1, ny, nz, ncol, nb, true, true).total
                                  : SlabLayout<float>(1, ny, nz, ncol, nb, true, true).total;
  return least <= kSlabRoom;
}

bool active(const jrg_plan* P) { return P->cols && jrg_fast_paths(-1) == 1; }

template <typename R> static int launch_columns(const jrg_plan* P, int op, const fast::Args& a, cudaStream_t st) {
  switch (P->nx) {
#define CASE(N) case N: return run_columns<R, N>(P, op, a, st);
    JRG_COLS_SIZES(CASE)
#undef CASE
    default: return 0;
  }
}

template <typename R> int dispatch(const jrg_plan* P, int op, const fast::Args& a, cudaStream_t st) {
  if ((op == fast::OP_LINE_DENSITY || op == fast::OP_LINE_APPLY_V) && P->nx == P->ny && P->ny == P->nz) {
    switch (P->nx) {
#define CASE(N) case N: if (cube_used<R, N>()) return run_cube<R, N>(P, op, a, st); break;
      JRG_COLS_SIZES(CASE)
#undef CASE
      default: break;
    }
  }
  switch (op) {
    case fast::OP_LINE_DENSITY: return launch_density<R>(P, a, st);
    case fast::OP_LINE_APPLY_V: return launch_apply<R>(P, a, st);
    default: return launch_columns<R>(P, op, a, st);
  }
}
template int dispatch<float>(const jrg_plan*, int, const fast::Args&, cudaStream_t);
template int dispatch<double>(const jrg_plan*, int, const fast::Args&, cudaStream_t);

}  // namespace cols
}  // namespace jrg
