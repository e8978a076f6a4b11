// Line transforms of the slab kernels (see fft_cols.cuh): the y and z phases of a
// tile of bands.
#pragma once
#include "fft_cols.cuh"

namespace jrg {
namespace cols {

// y inverse of every (band, window z): columns of T -> m; halves: the odd ones in
// the upper part of the index, so that warps are uniform in the parity
template <typename C, int NY, int PZ> __device__ __forceinline__ void y_inverse_body(const Tile<C>& q) {
  using R = decltype(C::x);
  constexpr int H = win_half<NY>(), parts = halves<R, NY>() ? 2 : 1;
  const int pz = PZ > 0 ? PZ : q.pz, wz = PZ > 0 ? PZ : q.wz;   // a fixed pitch is an odd window's
#pragma unroll 1
  for (int l = threadIdx.x; l < parts * q.n * wz; l += blockDim.x) {
    const int pt = l / wz, zc = l - pt * wz;
    const int par = parts == 2 && pt >= q.n ? 1 : 0, t = pt - par * q.n;
    const C* src = q.src + (size_t)shared_at<unsigned short>(q.list)[t] * q.bstride;
    C* dst = shared_at<C>(q.m) + t * NY * pz + zc;
    const short* col = shared_at<short>(q.col) + zc;
    auto load = [&](auto ii) {
      const int c = col[win_pos<NY, H>(ii.value) * wz];
      return c >= 0 ? src[c] : czero<C>();
    };
    if constexpr (parts == 2) {
      dst += par * pz;
      ln::half_inverse<C, NY, H>(par, load, [&](auto kk, C v) { dst[2 * kk.value * pz] = v; });
    } else {
      line_fft<C, NY, +1, H>(load, [&](auto kk, C v) { dst[kk.value * pz] = v; });
    }
  }
}

// y forward of every (band, window z).  Whole lines go straight to the columns of
// T; halves leave E[q] in row 2q and O'[q] in row 2q + 1 of m, their own places.
template <typename C, int NY, int PZ> __device__ __forceinline__ void y_forward_body(const Tile<C>& q) {
  using R = decltype(C::x);
  constexpr int H = win_half<NY>(), parts = halves<R, NY>() ? 2 : 1;
  const int pz = PZ > 0 ? PZ : q.pz, wz = PZ > 0 ? PZ : q.wz;   // a fixed pitch is an odd window's
#pragma unroll 1
  for (int l = threadIdx.x; l < parts * q.n * wz; l += blockDim.x) {
    const int pt = l / wz, zc = l - pt * wz;
    const int par = parts == 2 && pt >= q.n ? 1 : 0, t = pt - par * q.n;
    C* m = shared_at<C>(q.m) + t * NY * pz + zc;
    if constexpr (parts == 2) {
      m += par * pz;
      ln::half_forward<C, NY>(par, [&](auto ii) { return m[2 * ii.value * pz]; },
                              [&](auto kk, C v) { m[2 * kk.value * pz] = v; });
    } else {
      C* dst = q.src + (size_t)shared_at<unsigned short>(q.list)[t] * q.bstride;
      const short* col = shared_at<short>(q.col) + zc;
      line_fft<C, NY, -1, -1>([&](auto ii) { return m[ii.value * pz]; },
                              [&](auto kk, C v) {
                                if constexpr (in_win<NY, H>(kk.value)) {
                                  const int c = col[win_pos<NY, H>(kk.value) * wz];
                                  if (c >= 0) dst[c] = v;
                                }
                              });
    }
  }
}

template <typename C, int NY> __device__ void y_inverse(Tile<C> q) { y_inverse_body<C, NY, 0>(q); }
template <typename C, int NY> __device__ void y_forward(Tile<C> q) { y_forward_body<C, NY, 0>(q); }

// z inverse of every (band, y) and sum of w |psi|^2 into the slab's sums (share s
// of sub takes every sub-th band; the shares add up one after the other)
template <typename C, int NZ>
__device__ void z_density(Tile<C> q, int sw_at, int sum_at, int ny, int pv, int sub) {
  using R = decltype(C::x);
  const R* sw = shared_at<R>(sw_at);
  R* sum = shared_at<R>(sum_at);
  const unsigned short* list = shared_at<unsigned short>(q.list);
  constexpr int H = win_half<NZ>(), parts = halves<R, NZ>() ? 2 : 1, M = NZ / parts;
  const int s = threadIdx.x / (parts * ny), yp = threadIdx.x - s * (parts * ny);
  const int par = yp / ny, y = yp - par * ny;
  R acc[M];
#pragma unroll
  for (int k = 0; k < M; ++k) acc[k] = (R)0;
  if (s < sub) {
#pragma unroll 1
    for (int t = s; t < q.n; t += sub) {
      const C* row = shared_at<C>(q.m) + (t * ny + y) * q.pz;
      const R w = sw[list[t]];
      auto load = [&](auto ii) { return row[win_pos<NZ, H>(ii.value)]; };
      auto store = [&](auto kk, C v) { acc[kk.value] += w * (v.x * v.x + v.y * v.y); };
      if constexpr (parts == 2) ln::half_inverse<C, NZ, H>(par, load, store);
      else line_fft<C, NZ, +1, H>(load, store);
    }
  }
#pragma unroll 1
  for (int p = 0; p < sub; ++p) {
    if (p) __syncthreads();
    if (s == p) {
      R* d = sum + y * pv + par;
#pragma unroll
      for (int k = 0; k < M; ++k) d[parts * k] += acc[k];
    }
  }
}

// z inverse, times V, z forward of every (band, y), in place in the window row;
// halves: the even z, whose forward half is kept, then the odd z
template <typename C, int NZ, int PZ>
__device__ __forceinline__ void z_apply_body(const Tile<C>& q, int sv_at, int ny, int pv, int sub) {
  using R = decltype(C::x);
  const R* sv = shared_at<R>(sv_at);
  constexpr int H = win_half<NZ>();
  const int s = threadIdx.x / ny, y = threadIdx.x - s * ny;
  if (s >= sub) return;
  const R* vrow = sv + y * pv;
#pragma unroll 1
  for (int t = s; t < q.n; t += sub) {
    C* row = shared_at<C>(q.m) + (t * ny + y) * (PZ > 0 ? PZ : q.pz);
    auto load = [&](auto ii) { return row[win_pos<NZ, H>(ii.value)]; };
    if constexpr (halves<R, NZ>()) {
      constexpr int M = NZ / 2;
      C ev[M];
#pragma unroll 1
      for (int par = 0; par < 2; ++par) {
        C v[M], o[M];
        ln::half_inverse<C, NZ, H>(par, load, [&](auto kk, C a) {
          v[kk.value] = cscale(a, vrow[2 * kk.value + par]);
        });
        ln::half_forward<C, NZ>(par, [&](auto ii) { return v[ii.value]; },
                                [&](auto kk, C a) { o[kk.value] = a; });
        if (par == 0) {
#pragma unroll
          for (int k = 0; k < M; ++k) ev[k] = o[k];
        } else {
          ln::sfor<M>([&](auto kk) {
            constexpr int k = kk.value;
            if constexpr (in_win<NZ, H>(k)) row[win_pos<NZ, H>(k)] = ln::vadd(ev[k], o[k]);
            if constexpr (in_win<NZ, H>(k + M)) row[win_pos<NZ, H>(k + M)] = ln::vsub(ev[k], o[k]);
          });
        }
      }
    } else {
      C v[NZ];
      line_fft<C, NZ, +1, H>(load, [&](auto kk, C a) { v[kk.value] = cscale(a, vrow[kk.value]); });
      line_fft<C, NZ, -1, -1>([&](auto ii) { return v[ii.value]; },
                              [&](auto kk, C a) {
                                if constexpr (in_win<NZ, H>(kk.value)) row[win_pos<NZ, H>(kk.value)] = a;
                              });
    }
  }
}

// The same for lengths by halves with the two halves of a line on two threads
// (different warps): the odd half leaves its O' in the window row, which every
// thread has read by then, and the even half adds its E.  Half the registers of a
// thread that keeps E while it does the odd half: twelve warps on an SM instead of
// six (96^3, 160 bands: 5.02 ms before).  All threads of the CTA call it.
template <typename C, int NZ, int PZ>
__device__ __forceinline__ void z_apply_pairs(const Tile<C>& q, int sv_at, int pv, int sub) {
  using R = decltype(C::x);
  constexpr int H = win_half<NZ>(), M = NZ / 2;
  const int s = threadIdx.x / (2 * NZ), yp = threadIdx.x - s * (2 * NZ);
  const int par = yp / NZ, y = yp - par * NZ;
  const R* vrow = shared_at<R>(sv_at) + y * pv + par;
#pragma unroll 1
  for (int t0 = 0; t0 < q.n; t0 += sub) {
    const bool act = s < sub && t0 + s < q.n;
    C* row = shared_at<C>(q.m) + ((act ? t0 + s : 0) * NZ + y) * PZ;
    C o[M];
    if (act) {
      C v[M];
      ln::half_inverse<C, NZ, H>(par, [&](auto ii) { return row[win_pos<NZ, H>(ii.value)]; },
                                 [&](auto kk, C a) { v[kk.value] = cscale(a, vrow[2 * kk.value]); });
      ln::half_forward<C, NZ>(par, [&](auto ii) { return v[ii.value]; }, [&](auto kk, C a) { o[kk.value] = a; });
    }
    __syncthreads();
    if (act && par) {
      ln::sfor<M>([&](auto kk) {
        constexpr int k = kk.value;
        if constexpr (in_win<NZ, H>(k)) row[win_pos<NZ, H>(k)] = o[k];
        if constexpr (in_win<NZ, H>(k + M)) row[win_pos<NZ, H>(k + M)] = ln::cneg(o[k]);
      });
    }
    __syncthreads();
    if (act && !par) {
      ln::sfor<M>([&](auto kk) {
        constexpr int k = kk.value;
        if constexpr (in_win<NZ, H>(k)) row[win_pos<NZ, H>(k)] = ln::vadd(o[k], row[win_pos<NZ, H>(k)]);
        if constexpr (in_win<NZ, H>(k + M)) row[win_pos<NZ, H>(k + M)] = ln::vadd(o[k], row[win_pos<NZ, H>(k + M)]);
      });
    }
  }
}

template <typename C, int NZ>
__device__ void z_apply(Tile<C> q, int sv, int ny, int pv, int sub) {
  z_apply_body<C, NZ, 0>(q, sv, ny, pv, sub);
}

}  // namespace cols
}  // namespace jrg
