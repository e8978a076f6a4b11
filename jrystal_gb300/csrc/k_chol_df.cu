// Cholesky factor and inverse of the Gram matrices of the FP32 path, in
// double-float arithmetic on the FP32 pipes.
//
// FP64 arithmetic runs at 1/64 of the FP32 rate on this GPU, and a 160-band
// Cholesky + triangular inverse is ~5.5 million complex multiply-adds per
// (s,k) block, one CTA each; in FP64 through global memory that took 3.1 ms
// for the nine blocks of the 64-atom cell.  Here each block's upper triangle
// lives in shared memory (packed rows, 16 bytes per complex entry: 206 KB at
// 160 bands) as double-float pairs (hi + lo, about 48 significant bits: the
// Dekker/Knuth error-free transformations TwoSum and TwoProd, the latter with
// an FMA), and both the factorisation and the inversion take one barrier per
// pivot (256 threads up to 64 bands, 1024 above; the FP64 element-parallel
// kernel takes more bands than the shared memory holds):
//   factorisation (R^H R = S, R upper): at pivot k every thread reads the
//     unscaled pivot d_k = U[k][k] and updates U[i][j] -= conj(U[k][i])
//     U[k][j] / d_k for k < i <= j (one warp per row, lanes along j); the rows
//     are scaled by 1/sqrt(d_k) once at the end;
//   inversion (X = R^{-1}, in place, bottom-up): location (k, j > k) holds
//     a_kj = -sum_{l > k} R[k][l] X[l][j] when pivot k is reached, so
//     X[k][j] = a_kj / R[k][k] and X[k][k] = 1 / R[k][k]; the rows i < k are
//     updated with X[i][j] -= R[i][k] X[k][j] (j > k) and X[i][k] = -R[i][k] X[k][k],
//     each warp reading R[i][k] before its lane j = k overwrites it; the
//     rows are scaled at the end.
// The chain of a pivot (its reciprocal, the scaled row entry, one update) bounds the
// kernel: 24 bands 43 -> 37 us and 160 bands 1.12 -> 0.93 ms with the update's
// products subtracted in one renormalisation, an approximate reciprocal refined in
// FP32 before the double-float step, the inverse square roots in parallel and
// 32-bit indices.
// A pivot d_k <= min_pivot * S_kk, or a non-finite one, sets the breakdown
// bit and is replaced by 1 (as the FP64 kernels do); the condition estimate
// max_k S_kk / d_k goes to the flag word.
#include "plan.h"

namespace jrg {

namespace dfa {

struct df { float hi, lo; };

__device__ __forceinline__ df from_d(double x) {
  const float h = (float)x;
  return {h, (float)(x - (double)h)};
}
__device__ __forceinline__ double to_d(df a) { return (double)a.hi + (double)a.lo; }
// s + e = a + b exactly (Knuth's TwoSum)
__device__ __forceinline__ df two_sum(float a, float b) {
  const float s = a + b, bb = s - a;
  return {s, (a - (s - bb)) + (b - bb)};
}
// |a| >= |b| (Dekker's Fast2Sum)
__device__ __forceinline__ df fast_two_sum(float a, float b) {
  const float s = a + b;
  return {s, b - (s - a)};
}
__device__ __forceinline__ df add(df a, df b) {
  df s = two_sum(a.hi, b.hi);
  s.lo += a.lo + b.lo;
  return fast_two_sum(s.hi, s.lo);
}
__device__ __forceinline__ df neg(df a) { return {-a.hi, -a.lo}; }
// product, the high part's rounding error recovered with an FMA
__device__ __forceinline__ df mul(df a, df b) {
  const float p = a.hi * b.hi;
  float e = fmaf(a.hi, b.hi, -p);
  e = fmaf(a.hi, b.lo, e);
  e = fmaf(a.lo, b.hi, e);
  return fast_two_sum(p, e);
}

struct dc { df re, im; };   // complex double-float

__device__ __forceinline__ dc ld(const float4* p) {
  const float4 v = *p;
  return {{v.x, v.y}, {v.z, v.w}};
}
__device__ __forceinline__ void st(float4* p, dc a) { *p = make_float4(a.re.hi, a.re.lo, a.im.hi, a.im.lo); }
__device__ __forceinline__ dc cscale(dc a, df s) { return {mul(a.re, s), mul(a.im, s)}; }
__device__ __forceinline__ dc conj(dc a) { return {a.re, neg(a.im)}; }

// c - a b with one renormalisation: the products' and sums' rounding errors are
// collected in the low part (56 operations a complex element, 72 as a product and
// a difference of double-floats)
__device__ __forceinline__ df sub2(df c, df a, df b, float sg, df x, df y) {
  // c - a b - sg x y, sg = +-1
  const float p = a.hi * b.hi, q = sg * x.hi * y.hi;
  float e = fmaf(a.hi, b.hi, -p), f = fmaf(sg * x.hi, y.hi, -q);
  e = fmaf(a.lo, b.hi, fmaf(a.hi, b.lo, e));
  f = fmaf(sg * x.lo, y.hi, fmaf(sg * x.hi, y.lo, f));
  const df s = two_sum(c.hi, -p), t = two_sum(s.hi, -q);
  return fast_two_sum(t.hi, ((s.lo + t.lo) + c.lo) - (e + f));
}
__device__ __forceinline__ dc submul(dc c, dc a, dc b) {
  return {sub2(c.re, a.re, b.re, -1.f, a.im, b.im), sub2(c.im, a.re, b.im, 1.f, a.im, b.re)};
}

// 1 / x for x > 0: approximate reciprocal, one Newton step in FP32 and one in
// double-float.  The approximate division returns 0 above 2^126.
__device__ __forceinline__ df recip(df x) {
  float r0 = x.hi > 0x1p126f ? 1.0f / x.hi : __fdividef(1.0f, x.hi);
  r0 = fmaf(r0, fmaf(-x.hi, r0, 1.0f), r0);
  // e = 1 - x r0, r = r0 + r0 e
  const df xr = mul(x, df{r0, 0.f});
  const df e = add(df{1.0f, 0.f}, neg(xr));
  return add(df{r0, 0.f}, mul(df{r0, 0.f}, e));
}

}  // namespace dfa


__host__ __device__ inline size_t chol_df_smem(int nb) {
  return (size_t)nb * (nb + 1) / 2 * sizeof(float4) + (size_t)nb * (sizeof(double) + 3 * sizeof(float));
}

// the 1/sqrt of the FP64 kernels (FP32 seed, three Newton steps in FP64)
__device__ __forceinline__ double rsqrt_nr(double d) {
  double r = (double)rsqrtf((float)d);
  r = r * (1.5 - 0.5 * d * r * r);
  r = r * (1.5 - 0.5 * d * r * r);
  r = r * (1.5 - 0.5 * d * r * r);
  return r;
}

template <int NT>
__global__ void __launch_bounds__(NT, 1)
k_cholesky_inv_df(const double2* __restrict__ S, double2* __restrict__ Ri, int nb, int* __restrict__ flags,
                  double min_pivot, int nsplit) {
  using namespace dfa;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // FP64 work stays off the per-element paths (1/64 of the FP32 rate): the
  // pivot test compares FP32 values, pivots and their inverse square roots
  // are kept as double-float pairs, and one lane per row forms 1/sqrt(d_k)
  float4* U = reinterpret_cast<float4*>(smem_raw);                         // packed upper rows
  double* sdiag = reinterpret_cast<double*>(U + (size_t)nb * (nb + 1) / 2);  // S_kk
  float* thr = reinterpret_cast<float*>(sdiag + nb);                        // min_pivot S_kk
  df* dpiv = reinterpret_cast<df*>(thr + nb);                               // d_k, then 1/sqrt(d_k)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = NT / 32;
  const size_t off = (size_t)blockIdx.x * nb * nb;
  auto idx = [nb](int i, int j) { return i * (2 * nb - i - 1) / 2 + j; };
  // upper triangle of the Hermitian part of S, the sum of nsplit parts
  const double2* s0 = S + off * nsplit;
  for (int i = warp; i < nb; i += nwarp)
    for (int j = i + lane; j < nb; j += 32) {
      double2 a = s0[i * nb + j], b = s0[j * nb + i];
      for (int p = 1; p < nsplit; ++p) {
        const double2 u = s0[p * nb * nb + i * nb + j], v = s0[p * nb * nb + j * nb + i];
        a.x += u.x; a.y += u.y; b.x += v.x; b.y += v.y;
      }
      const double re = 0.5 * (a.x + b.x), im = i == j ? 0.0 : 0.5 * (a.y - b.y);
      st(U + idx(i, j), dc{from_d(re), from_d(im)});
      if (i == j) { sdiag[i] = a.x; thr[i] = (float)(min_pivot * a.x); }
    }
  __syncthreads();
  // factorisation with unscaled pivot rows
  bool broke = false;
  for (int k = 0; k < nb; ++k) {
    df d = ld(U + idx(k, k)).re;
    if (!(d.hi > thr[k]) || !isfinite(d.hi)) { d = df{1.0f, 0.f}; broke = true; }
    const df invd = recip(d);
    for (int i = k + 1 + warp; i < nb; i += nwarp) {
      const dc a = cscale(conj(ld(U + idx(k, i))), invd);   // conj(U[k][i]) / d_k
      for (int j = i + lane; j < nb; j += 32) {
        float4* p = U + idx(i, j);
        st(p, submul(ld(p), a, ld(U + idx(k, j))));
      }
    }
    if (tid == 0) dpiv[k] = d;
    __syncthreads();
  }
  if (broke && tid == 0) atomicOr(flags, 1);
  // 1/sqrt(d_k) and sqrt(d_k), a thread each (one lane per row in turn put the FP64
  // chain of every row on the path), then row k scaled: R
  for (int k = tid; k < nb; k += NT) {
    const double dk = to_d(dpiv[k]), rs = rsqrt_nr(dk);
    dpiv[k] = from_d(rs);
    st(U + idx(k, k), dc{from_d(dk * rs), df{0.f, 0.f}});
  }
  __syncthreads();
  for (int k = warp; k < nb; k += nwarp) {
    const df s = dpiv[k];
    for (int j = k + 1 + lane; j < nb; j += 32) {
      float4* p = U + idx(k, j);
      st(p, cscale(ld(p), s));
    }
  }
  __syncthreads();
  // inversion in place, bottom-up
  for (int k = nb - 1; k >= 0; --k) {
    const df dk = dpiv[k];   // 1 / R[k][k] = X[k][k]
    for (int i = warp; i < k; i += nwarp) {
      const dc r = ld(U + idx(i, k));   // R[i][k]
      __syncwarp();                     // every lane has R[i][k] before lane j = k overwrites it
      for (int j = k + lane; j < nb; j += 32) {
        float4* p = U + idx(i, j);
        if (j == k) {
          st(p, cscale(r, neg(dk)));
        } else {
          const dc xkj = cscale(ld(U + idx(k, j)), dk);   // X[k][j] = a_kj / R[k][k]
          st(p, submul(ld(p), r, xkj));
        }
      }
    }
    __syncthreads();
  }
  // X[k][j] = a_kj / R[k][k] (j > k), X[k][k] = 1 / R[k][k]; lower part zero
  for (int i = warp; i < nb; i += nwarp) {
    const df di = dpiv[i];
    for (int j = lane; j < nb; j += 32) {
      double2 v = make_double2(0.0, 0.0);
      if (j == i) v = make_double2(to_d(di), 0.0);
      else if (j > i) {
        const dc x = cscale(ld(U + idx(i, j)), di);
        v = make_double2(to_d(x.re), to_d(x.im));
      }
      Ri[off + (size_t)i * nb + j] = v;
    }
  }
  // condition estimate off the pivot chain: S_kk / d_k = S_kk (1/sqrt(d_k))^2
  if (warp == 0) {
    double c = 0.0;
    for (int k = lane; k < nb; k += 32) {
      const double r = to_d(dpiv[k]);
      c = fmax(c, fabs(sdiag[k]) * r * r);
    }
    for (int o = 16; o > 0; o >>= 1) c = fmax(c, __shfl_xor_sync(0xffffffffu, c, o));
    if (lane == 0) {
      double est = broke ? __longlong_as_double(0x7ff0000000000000LL) : c;
      if (!(est >= 0.0)) est = __longlong_as_double(0x7ff0000000000000LL);
      atomicMax(reinterpret_cast<unsigned long long*>(flags + 2), (unsigned long long)__double_as_longlong(est));
    }
  }
}

// 1: launched; 0: the triangle does not fit in shared memory (use the FP64
// kernel); < 0: -status
int launch_cholesky_inv_df(const double2* S, double2* Ri, int nsk, int nb, int* flags, double min_pivot,
                           cudaStream_t st, int nsplit) {
  const size_t sm = chol_df_smem(nb);
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 0;
  if (sm > (size_t)optin) return 0;
  // one warp per row of the update: 8 warps up to 64 bands, 32 above
  auto go = [&](auto kern, int nt) -> cudaError_t {
    cudaError_t e = allow_smem((const void*)kern, sm);
    if (e != cudaSuccess) return e;
    kern<<<nsk, nt, sm, st>>>(S, Ri, nb, flags, min_pivot, nsplit);
    return cudaSuccess;
  };
  cudaError_t e = nb <= 64 ? go(k_cholesky_inv_df<256>, 256) : go(k_cholesky_inv_df<1024>, 1024);
  if (e != cudaSuccess) return -cuda_fail(e, "cudaFuncSetAttribute(k_cholesky_inv_df)");
  count_launch();
  e = cudaGetLastError();
  if (e != cudaSuccess) return -cuda_fail(e, "k_cholesky_inv_df");
  return 1;
}

}  // namespace jrg
