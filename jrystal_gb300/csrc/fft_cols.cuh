// Column-first transforms between the plane-wave sphere and the real grid.
//
// The inverse transform runs x first, on the (y, z) columns that the sphere
// touches, then y and z of each x slab with the slab's consumer fused in
// (density, or times V(r) and back).  The intermediate between the two passes
// is T[band][x][column], i.e. only the sphere's (y, z) disk: a fifth of the grid
// (64^3: 797 of 4096 columns), where planes transformed in y and z hold nact/nx,
// about half.  Every line is transformed by one thread in registers
// (fft_line.cuh), so that any two axis lengths combine: the slab kernels take
// the lengths at run time and switch into one function per length and phase.
//
//   k_cols_inv       sphere -> T      (x inverse, one thread per column)
//   k_slab_density   T -> density     (y inverse, z inverse, sum w |psi|^2)
//   k_slab_apply_v   T -> T in place  (y, z inverse, times V, z, y forward)
//   k_cols_fwd       T -> g_C         (x forward, kinetic term, weights)
//
// Before, the planes of each band were transformed in y and z first, by several
// threads a line with a shared-memory exchange in every transform: 0.99 ms for the
// four passes at the Si8 64^3 workload (27 k-points, 24 bands, FP32), now 0.55 ms;
// at 96^3 (160 bands) 12.9, now 6.4 ms; 30 x 45 x 64 (84 bands) 444, now 146 us.
//
// Every active index of the sphere lies in the alias-free window |i| < N/4 of its
// axis; spheres that reach further keep the plane-first kernels (k_fft_fast.cu,
// k_fft.cu).  Bands of weight zero are left out: they add nothing to the density
// and have no gradient (a caller's non-finite coefficients in such a band still
// reach the density, see density_entry in capi.cu).
#pragma once
#include <algorithm>
#include <type_traits>

#include "fast_dispatch.h"
#include "fft_line.cuh"
#include "plan.h"

namespace jrg {
namespace cols {

using ln::in_win;
using ln::line_fft;
using ln::win_half;
using ln::win_pos;

template <int N> __host__ __device__ constexpr int win_n() { return 2 * win_half<N>() + 1; }
inline __host__ __device__ int window(int n) { return 2 * ((n - 1) / 4) + 1; }

// axis lengths with kernels: the products of 2, 3, 5, 7 from 16 to 96 (75 and 81,
// odd and too long for the registers, keep the plane-first kernels)
#define JRG_COLS_SIZES_0(F) F(16) F(18) F(20) F(21) F(24) F(25) F(27) F(28) F(30) F(32) F(35) F(36)
#define JRG_COLS_SIZES_1(F) F(40) F(42) F(45) F(48) F(49) F(50) F(54)
#define JRG_COLS_SIZES_2(F) F(56) F(60) F(63) F(64) F(70)
#define JRG_COLS_SIZES_3(F) F(72) F(80) F(84) F(90) F(96)
#define JRG_COLS_SIZES(F) JRG_COLS_SIZES_0(F) JRG_COLS_SIZES_1(F) JRG_COLS_SIZES_2(F) JRG_COLS_SIZES_3(F)

// Lines by halves (fft_line.cuh) or whole in one thread.  A whole FP32 line of 64
// needs 128 registers and the least instructions; longer ones, and FP64 lines
// above 32, spill.
template <typename R, int N> __host__ __device__ constexpr bool halves() {
  return N % 2 == 0 && N > (sizeof(R) == 4 ? 64 : 32);
}
template <typename R> __host__ __device__ inline int parts_of(int n) {
  return n % 2 == 0 && n > (sizeof(R) == 4 ? 64 : 32) ? 2 : 1;
}

// Registers: 168 a thread for the adjoint pass (384 threads on an SM), 255 for
// the density pass, whose threads keep their line's sums.
constexpr int kApplyThreads = 384;
constexpr int kDensityThreads = 256;
constexpr int kSlabMost = 128;      // threads of a slab CTA as launched
constexpr size_t kSlabRoom = 226 * 1024;   // shared memory of a CTA, its few static words aside

// ---- shared memory: the one description that launch and kernel use ---------------
template <typename R> struct SlabLayout {
  size_t grid, pos, col, w, list, total;
  int pz, pv;
  // tile planes [ny][pz], a real slab [ny][pv] (V, or the density sums), places of
  // the columns, column map, weights, band list
  __host__ __device__ SlabLayout(int tile, int ny, int nz, int ncol, int bands, bool weights, bool places) {
    pz = window(nz) | 1;            // odd: rows and columns both free of bank conflicts
    pv = nz | 1;
    size_t o = 0;
    auto take = [&o](size_t bytes) { const size_t r = o; o += (bytes + 15) / 16 * 16; return r; };
    take(sizeof(C_t<R>) * (size_t)tile * ny * pz);
    grid = take(sizeof(R) * (size_t)ny * pv);
    pos = take(places ? sizeof(int) * (size_t)ncol : 0);
    col = take(sizeof(short) * (size_t)window(ny) * window(nz));
    w = take(weights ? sizeof(R) * (size_t)bands : 0);
    list = take(sizeof(unsigned short) * (size_t)bands);
    total = o;
  }
};

// Bands of the group [b_begin, b_end) with a non-zero weight, in order, into list
// (by warp 0; the caller synchronises).
__device__ __forceinline__ void live_bands(const double* __restrict__ w, int b_begin, int b_end,
                                           unsigned short* list, int* count) {
  if (threadIdx.x >= 32) return;
  int n = 0;
  for (int b0 = b_begin; b0 < b_end; b0 += 32) {
    const int b = b0 + threadIdx.x;
    const bool live = b < b_end && w[b] != 0.0;
    const unsigned m = __ballot_sync(0xffffffffu, live);
    if (live) list[n + __popc(m & ((1u << threadIdx.x) - 1))] = (unsigned short)(b - b_begin);
    n += __popc(m);
  }
  if (threadIdx.x == 0) *count = n;
}

// The columns of the next tile into L2 while this one is transformed.
template <typename C>
__device__ __forceinline__ void prefetch_tile(const C* src, const unsigned short* list, int n, int tp,
                                              size_t band_stride) {
  const int lines = (tp * (int)sizeof(C) + 127) / 128;
  for (int i = threadIdx.x; i < n * lines; i += blockDim.x) {
    const int t = i / lines;
    const char* p = reinterpret_cast<const char*>(src + (size_t)list[t] * band_stride) + (i - t * lines) * 128;
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
  }
}

// What the phases of one tile work on.  Places in shared memory are byte offsets
// into it, so that the phase functions address shared memory as such.
template <typename C> struct Tile {
  C* src;           // T of the group's first band at this x
  size_t bstride;   // elements from band to band
  int n;            // bands of the tile
  int list;         // [n] band of the group
  int m;            // planes [n][ny][pz]
  int col;          // [window y][window z] column, or -1
  int wz, pz;
};
template <typename T> __device__ __forceinline__ T* shared_at(int offset) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  return reinterpret_cast<T*>(smem_raw + offset);
}

// The column map into shared memory and, with places, where a column's y forward
// output stands in the planes: row 2q of E[q], q = k mod ny/2 (O'[q] one row
// below), and the sign of O'[q] in the lowest bit.
template <bool PLACES>
__device__ __forceinline__ void column_places(const short* __restrict__ col_of, short* scol, int* spos, int ny, int wy,
                                              int wz, int pz) {
  for (int i = threadIdx.x; i < wy * wz; i += blockDim.x) {
    const int c = col_of[i];
    scol[i] = (short)c;
    if (PLACES && c >= 0) {
      const int yc = i / wz, zc = i - yc * wz;
      const int k = yc <= (ny - 1) / 4 ? yc : yc + (ny - wy);
      spos[c] = 2 * (2 * (k % (ny / 2)) * pz + zc) + (k >= ny / 2 ? 1 : 0);
    }
  }
}

// E[q] +- O'[q] of each column back into T
template <typename C>
__device__ __forceinline__ void columns_back(const Tile<C>& q, const unsigned short* list, const int* spos, int ncol,
                                             int ny, int pz) {
#pragma unroll 1
  for (int t = 0; t < q.n; ++t) {
    C* dst = q.src + (size_t)list[t] * q.bstride;
    const C* m = shared_at<C>(q.m) + t * ny * pz;
    for (int c = threadIdx.x; c < ncol; c += blockDim.x) {
      const int p = spos[c];
      const C e = m[p >> 1], o = m[(p >> 1) + pz];
      dst[c] = (p & 1) ? ln::vsub(e, o) : ln::vadd(e, o);
    }
  }
}

// The phases of a tile, one function per length.  They are compiled by length in
// several translation units (cols_lines.cuh, k_cols_part.cu) and linked into the
// slab kernels as device functions.
template <typename C, int NY> __device__ __noinline__ void y_inverse(Tile<C> q);
template <typename C, int NY> __device__ __noinline__ void y_forward(Tile<C> q);
template <typename C, int NZ>
__device__ __noinline__ void z_density(Tile<C> q, int sw, int sum, int ny, int pv, int sub);
template <typename C, int NZ>
__device__ __noinline__ void z_apply(Tile<C> q, int sv, int ny, int pv, int sub);

// ---- host side ------------------------------------------------------------------
// same return convention as fast::dispatch: 1 launched, 0 not covered, < 0: -status
inline int launched(const char* what) {
  count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 1 : -cuda_fail(e, what);
}
inline int prep(const void* kernel, size_t bytes) {
  cudaError_t e = allow_smem(kernel, bytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                             (int)cudaSharedmemCarveoutMaxShared);
  return e == cudaSuccess ? 1 : -cuda_fail(e, "cudaFuncSetAttribute(column transforms)");
}

struct SlabShape { int threads = 0, tile = 0, sub = 0; size_t smem = 0; };

// Threads, bands per tile and bands in flight in the z phase of a slab kernel.
// zlines: threads of the z phase for one band, ylines: lines of the y phase for
// one band, regs_threads: threads that the registers of an SM hold.  Of the shapes
// that leave few lanes idle over both phases, one with two CTAs on an SM and eight
// warps or more (adjoint pass at 64^3, us: 128 threads x 4 bands 258, 192 x 6
// 259, 256 x 8 284, 64 x 2 317, 128 x 2 326; at 48^3: 96 x 4 56, 96 x 2 75, 64 x
// 2 75).
template <class Bytes>
SlabShape slab_shape(int zlines, int ylines, int bands, int regs_threads, Bytes&& bytes) {
  SlabShape best;
  double best_cost = 1e30;
  for (int t = 64; t <= (zlines > 64 ? regs_threads : kSlabMost); t += 32) {
    const int sub = t / zlines;
    if (sub < 1) continue;
    for (int tile = 1; tile <= 24 && tile <= std::max(1, bands); ++tile) {
      const size_t sm = bytes(tile);
      if (sm > kSlabRoom) break;
      const int ctas = std::min({regs_threads / t, (int)(227 * 1024 / (sm + 1024)), 24});
      const int warps = ctas * t / 32;
      const int steps = (bands + tile - 1) / tile;
      const double passes = (double)((tile * ylines + t - 1) / t) + (double)((tile + sub - 1) / sub) + 0.1;
      double cost = steps * (double)t * passes / bands;
      if (warps < 8) cost *= 1.0 + 0.08 * (8 - warps);
      if (ctas < 2) cost *= 1.1;
      if (ctas > 2) cost *= 1.0 + 0.02 * (ctas - 2);   // more phases at once: more code in flight
      if (cost < best_cost - 1e-9) {
        best_cost = cost;
        best.threads = t; best.tile = tile; best.sub = std::min(sub, tile); best.smem = sm;
      }
    }
  }
  return best;
}

// Cubic grids have slab kernels of their own (k_cube.cuh) at every length, FP64 up to
// 63 points: above, lines by halves spill with the phases inlined (energy and gradient
// of 48 bands: 70^3 4460 us, 4417 with the phases as functions; 72^3 3766 and 3732).
// FP64 at 32^3 and 64^3 keeps the plane-first kernels (covers, k_fft_cols.cu).
template <typename R, int N> __host__ __device__ constexpr bool cube_used() {
  return sizeof(R) == 4 || (N != 32 && N <= 63);
}
template <typename R, int N> int run_cube(const jrg_plan* P, int op, const fast::Args& a, cudaStream_t st);
template <typename R, int N> int run_columns(const jrg_plan* P, int op, const fast::Args& a, cudaStream_t st);

}  // namespace cols
}  // namespace jrg
