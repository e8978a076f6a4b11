// One-thread line FFTs of compile-time length.
//
// A thread holds a whole line in registers: no exchange through shared
// memory, no barrier, no twiddle table.  The transform is a mixed-radix
// decimation in time, N = P*Q recursively down to radices 2, 3, 4, 5, 7 and
// 8, fully unrolled; twiddles are compile-time constants (FP32: the
// norm-balanced pair of common.cuh's balanced_twiddle, and hi + lo where no pair of
// floats comes near norm one).
//
// WIN: the half width H of the window of non-zero inputs (|i| <= H, counted
// cyclically; H < 0: every input).  The additions of the known zeros are left
// out at compile time (IEEE signed zeros keep the compiler from doing it
// itself).  Outputs that a caller's store functor drops are removed as dead
// code, which prunes the last stage the same way.
#pragma once
#include "common.cuh"
#include "fft_reg.cuh"

namespace jrg {
namespace ln {

using reg::cos2pi;
using reg::sfor;
using reg::sin2pi;

// widest alias-free window of a line: |i| < N/4
template <int N> __host__ __device__ constexpr int win_half() { return (N - 1) / 4; }
template <int N0, int H> __host__ __device__ constexpr bool in_win(int i) { return H < 0 || i <= H || i >= N0 - H; }
// position in the window (all of the line for H < 0), in line order
template <int N0, int H> __host__ __device__ constexpr int win_pos(int i) { return (H < 0 || i <= H) ? i : i - (N0 - 2 * H - 1); }

// ---- constants --------------------------------------------------------------
struct Pair32 { float c, s; };
__host__ __device__ constexpr double ulp32(double a) {          // spacing of the floats at |a|, a != 0
  if (a < 0) a = -a;
  double u = 1.1920928955078125e-07;        // 2^-23, the spacing in [1, 2)
  while (a < 1.0) { a *= 2.0; u *= 0.5; }
  return u;
}
__host__ __device__ constexpr double other32(double a) {        // the second-nearest float of a
  const float f = (float)a;
  if ((double)f == a) return a;
  return (double)f < a ? (double)f + ulp32(a) : (double)f - ulp32(a);
}
__host__ __device__ constexpr double abs_c(double a) { return a < 0 ? -a : a; }
__host__ __device__ constexpr Pair32 balanced32(double c, double s) {
  const double cs[2] = {(double)(float)c, other32(c)}, ss[2] = {(double)(float)s, other32(s)};
  int bi = 0, bj = 0;
  double be = abs_c(cs[0] * cs[0] + ss[0] * ss[0] - 1.0);
  for (int i = 0; i < 2; ++i)
    for (int j = 0; j < 2; ++j) {
      const double e = abs_c(cs[i] * cs[i] + ss[j] * ss[j] - 1.0);
      if (e < be) { be = e; bi = i; bj = j; }
    }
  return Pair32{(float)cs[bi], (float)ss[bj]};
}

// complex add and subtract: FP32 as one packed instruction on the register pair
// (add.rn.f32x2: the FP32 pipe's rate is the same, but it takes one issue slot
// instead of two, and issue slots are what bounds these transforms); the
// difference as fma(b, -1, a), exact like the subtraction
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ double2 vadd(double2 a, double2 b) { return cadd(a, b); }
__device__ __forceinline__ double2 vsub(double2 a, double2 b) { return csub(a, b); }

template <int DIR, typename C> __device__ __forceinline__ C rot90(C a) {   // DIR * i * a
  C r;
  if (DIR > 0) { r.x = -a.y; r.y = a.x; } else { r.x = a.y; r.y = -a.x; }
  return r;
}
template <typename C> __device__ __forceinline__ C cneg(C a) { a.x = -a.x; a.y = -a.y; return a; }

// a * exp(DIR 2 pi i K / N)
template <int DIR, int K, int N, typename C> __device__ __forceinline__ C twmul(C a) {
  constexpr int k = ((K % N) + N) % N;
  if constexpr (k == 0) return a;
  else if constexpr (4 * k == N) return rot90<DIR>(a);
  else if constexpr (2 * k == N) return cneg(a);
  else if constexpr (4 * k == 3 * N) return rot90<-DIR>(a);
  else {
    using R = decltype(a.x);
    constexpr double c = cos2pi(k, N), s = DIR * sin2pi(k, N);
    C r;
    if constexpr (sizeof(R) == 8) {
      r.x = fma(c, a.x, -s * a.y);
      r.y = fma(c, a.y, s * a.x);
    } else {
      if constexpr ((8 * k) % N == 0) {
        // odd multiples of pi/4, the only twiddles of the 8-point DFTs: sqrt(1/2)
        // as hi + lo (a pair rounded to float turns every transform by the same
        // angle, 1.5e-6 Ha per atom of external energy at the 64^3 Si8 cell)
        constexpr double m = c < 0 ? -c : c;
        constexpr float h = (float)m, l = (float)(m - (double)h);
        const float tx = (c < 0 ? -a.x : a.x) - (s < 0 ? -a.y : a.y);
        const float ty = (c < 0 ? -a.y : a.y) + (s < 0 ? -a.x : a.x);
        r.x = fmaf(h, tx, l * tx);
        r.y = fmaf(h, ty, l * ty);
      } else {
        constexpr Pair32 w = balanced32(c, s);
        if constexpr (9 * k == 2 * N || 9 * k == 7 * N) {
          // exp(+-2 pi i 2/9): the best pair is 4.6e-8 short of norm one (other ninths
          // 2.5e-8 at most), the sine as hi + lo makes it good
          constexpr float l = (float)(s - (double)w.s);
          r.x = fmaf(w.c, a.x, fmaf(-w.s, a.y, -l * a.y));
          r.y = fmaf(w.c, a.y, fmaf(w.s, a.x, l * a.x));
        } else {
          r.x = fmaf(w.c, a.x, -w.s * a.y);
          r.y = fmaf(w.c, a.y, w.s * a.x);
        }
      }
    }
    return r;
  }
}

template <bool ZA, bool ZB, typename C> __device__ __forceinline__ C addz(C a, C b) {
  if constexpr (ZB) return a;
  else if constexpr (ZA) return b;
  else return vadd(a, b);
}
template <bool ZA, bool ZB, typename C> __device__ __forceinline__ C subz(C a, C b) {
  if constexpr (ZB) return a;
  else if constexpr (ZA) return cneg(b);
  else return vsub(a, b);
}

// ---- base DFTs; bit i of M set: input i may be non-zero ----------------------
template <int N> __host__ __device__ constexpr bool is_base() { return N == 1 || N == 2 || N == 3 || N == 4 || N == 5 || N == 7 || N == 8; }

template <int N, int DIR, unsigned M, typename C> __device__ __forceinline__ void bdft(C (&v)[N]) {
  using R = decltype(v[0].x);
  if constexpr (N == 1 || M == 0) {
    return;
  } else if constexpr (N == 2) {
    constexpr bool z0 = !(M & 1), z1 = !(M & 2);
    const C a = v[0], b = v[1];
    v[0] = addz<z0, z1>(a, b);
    v[1] = subz<z0, z1>(a, b);
  } else if constexpr (N == 3) {
    constexpr bool z0 = !(M & 1), z1 = !(M & 2), z2 = !(M & 4);
    if constexpr (z1 && z2) {
      v[1] = v[0];
      v[2] = v[0];
    } else {
      constexpr double s3 = 0.86602540378443864676;
      const C t = addz<z1, z2>(v[1], v[2]);
      C d = subz<z1, z2>(v[1], v[2]);
      C m;
      if constexpr (z0) m = cscale(t, (R)-0.5);
      else { m.x = v[0].x - (R)0.5 * t.x; m.y = v[0].y - (R)0.5 * t.y; }
      if constexpr (sizeof(R) == 4) {
        // sqrt(3)/2 as hi + lo: a rounded constant scales the norm of every transform
        constexpr float h = (float)s3, l = (float)(s3 - (double)h);
        d.x = fmaf(h, d.x, l * d.x);
        d.y = fmaf(h, d.y, l * d.y);
      } else {
        d.x *= s3;
        d.y *= s3;
      }
      const C id = rot90<DIR>(d);
      v[0] = addz<z0, false>(v[0], t);
      v[1] = vadd(m, id);
      v[2] = vsub(m, id);
    }
  } else if constexpr (N == 4) {
    constexpr bool z0 = !(M & 1), z1 = !(M & 2), z2 = !(M & 4), z3 = !(M & 8);
    constexpr bool ze = z0 && z2, zo = z1 && z3;
    const C a = addz<z0, z2>(v[0], v[2]), b = subz<z0, z2>(v[0], v[2]);
    const C c = addz<z1, z3>(v[1], v[3]), d = rot90<DIR>(subz<z1, z3>(v[1], v[3]));
    v[0] = addz<ze, zo>(a, c);
    v[2] = subz<ze, zo>(a, c);
    v[1] = addz<ze, zo>(b, d);
    v[3] = subz<ze, zo>(b, d);
  } else if constexpr (N == 8) {
    constexpr unsigned E = (M & 1) | ((M >> 1) & 2) | ((M >> 2) & 4) | ((M >> 3) & 8);
    constexpr unsigned O = ((M >> 1) & 1) | ((M >> 2) & 2) | ((M >> 3) & 4) | ((M >> 4) & 8);
    C e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    bdft<4, DIR, E>(e);
    bdft<4, DIR, O>(o);
    sfor<4>([&](auto kk) {
      constexpr int k = kk.value;
      C t = o[k];
      if constexpr (O != 0) t = twmul<DIR, k, 8>(t);
      v[k] = addz<E == 0, O == 0>(e[k], t);
      v[k + 4] = subz<E == 0, O == 0>(e[k], t);
    });
  } else {
    // odd primes 5 and 7: sums and differences of the conjugate pairs
    constexpr int H = (N - 1) / 2;
    const C v0 = v[0];
    C t[H], d[H];
    sfor<H>([&](auto jj) {
      constexpr int j = jj.value + 1;
      constexpr bool za = !((M >> j) & 1), zb = !((M >> (N - j)) & 1);
      t[j - 1] = addz<za, zb>(v[j], v[N - j]);
      d[j - 1] = subz<za, zb>(v[j], v[N - j]);
    });
    C sum = v0;
    sfor<H>([&](auto jj) {
      constexpr int j = jj.value + 1;
      constexpr bool zp = !((M >> j) & 1) && !((M >> (N - j)) & 1);
      if constexpr (!zp) sum = vadd(sum, t[j - 1]);
    });
    v[0] = sum;
    sfor<H>([&](auto kk) {
      constexpr int k = kk.value + 1;
      C a = v0, b = czero<C>();
      // sin(2 pi/5) in FP32 as hi + lo: rounded to float it is 0.4 ulp off (the other
      // constants 0.28 at most), which scaled the density's norm by 9e-8 at 25^3 and
      // 60^3 and by 1.1e-7 at 50^3.  The lo product comes first: added to the finished
      // sum it would be rounded away.
      constexpr bool lo = sizeof(R) == 4 && N == 5;
      if constexpr (lo) b = cscale(d[k - 1], (R)(sin2pi(k * k, N) - (double)(float)sin2pi(k * k, N)));
      sfor<H>([&](auto jj) {
        constexpr int j = jj.value + 1;
        constexpr bool zp = !((M >> j) & 1) && !((M >> (N - j)) & 1);
        if constexpr (!zp) {
          constexpr R c = (R)cos2pi(j * k, N), s = (R)sin2pi(j * k, N);
          a.x = fma(c, t[j - 1].x, a.x);
          a.y = fma(c, t[j - 1].y, a.y);
          if constexpr (j == 1 && !lo) b = cscale(d[0], s);
          else { b.x = fma(s, d[j - 1].x, b.x); b.y = fma(s, d[j - 1].y, b.y); }
        }
      });
      const C ib = rot90<DIR>(b);
      v[k] = vadd(a, ib);
      v[N - k] = vsub(a, ib);
    });
  }
}

// outer radix of a composite length
template <int N> __host__ __device__ constexpr int outer_radix() {
  if (N == 16) return 4;
  if (N % 8 == 0) return 8;
  if (N % 4 == 0) return 4;
  if (N % 5 == 0) return 5;
  if (N % 3 == 0) return 3;
  if (N % 7 == 0) return 7;
  return 2;
}

// whether any of BASE + STRIDE*q (q < N) lies in the window, and the bit mask
template <int N, int N0, int H, int BASE, int STRIDE> __host__ __device__ constexpr unsigned win_mask() {
  unsigned m = 0;
  for (int q = 0; q < N; ++q)
    if (in_win<N0, H>(BASE + STRIDE * q)) m |= 1u << (q & 31);
  return m;
}

// DFT of the elements BASE + STRIDE*q (q < N) of the line, into out
template <int N, int DIR, int N0, int H, int BASE, int STRIDE, typename C, class L>
__device__ __forceinline__ void sub_fft(C (&out)[N], L& load) {
  if constexpr (is_base<N>()) {
    sfor<N>([&](auto qq) {
      constexpr int i = BASE + STRIDE * qq.value;
      if constexpr (in_win<N0, H>(i)) out[qq.value] = load(std::integral_constant<int, i>{});
      else out[qq.value] = czero<C>();
    });
    bdft<N, DIR, win_mask<N, N0, H, BASE, STRIDE>()>(out);
  } else {
    constexpr int P = outer_radix<N>(), Q = N / P;
    C y[P][Q];
    sfor<P>([&](auto pp) {
      sub_fft<Q, DIR, N0, H, BASE + STRIDE * pp.value, STRIDE * P>(y[pp.value], load);
    });
    sfor<Q>([&](auto kk) {
      constexpr int k = kk.value;
      C w[P];
      sfor<P>([&](auto pp) { w[pp.value] = twmul<DIR, pp.value * k, N>(y[pp.value][k]); });
      bdft<P, DIR, (1u << P) - 1>(w);
      sfor<P>([&](auto ss) { out[k + Q * ss.value] = w[ss.value]; });
    });
  }
}

// Whole line: load(integral_constant<i>) gives input i of the window, store(
// integral_constant<k>, value) takes output k (each output exactly once, as
// soon as it is formed).
template <typename C, int N, int DIR, int H, class L, class S>
__device__ __forceinline__ void line_fft(L&& load, S&& store) {
  if constexpr (is_base<N>()) {
    C v[N];
    sub_fft<N, DIR, N, H, 0, 1>(v, load);
    sfor<N>([&](auto kk) { store(kk, v[kk.value]); });
  } else {
    constexpr int P = outer_radix<N>(), Q = N / P;
    C y[P][Q];
    sfor<P>([&](auto pp) { sub_fft<Q, DIR, N, H, pp.value, P>(y[pp.value], load); });
    sfor<Q>([&](auto kk) {
      constexpr int k = kk.value;
      C w[P];
      sfor<P>([&](auto pp) { w[pp.value] = twmul<DIR, pp.value * k, N>(y[pp.value][k]); });
      bdft<P, DIR, (1u << P) - 1>(w);
      sfor<P>([&](auto ss) { store(std::integral_constant<int, k + Q * ss.value>{}, w[ss.value]); });
    });
  }
}

// ---- half lines ---------------------------------------------------------------
// A line of even length N over the window H as two transforms of M = N/2 points,
// so that half the registers hold it and both halves run the same code (par, the
// output or input parity, is a run-time value; only the twiddles of the odd half
// are behind a branch).  Inverse: output 2q + par is
//   sum_n (x[n] +- x[n + M]) w_N^(par n) W_M^(n q);
// inside the window |i| <= H < N/4 only one of the two summands is non-zero and no
// addition is left.  load(integral_constant<i>): input i of the window;
// store(integral_constant<q>, v): output 2q + par.
template <typename C, int N, int H, class L, class S>
__device__ __forceinline__ void half_inverse(int par, L&& load, S&& store) {
  static_assert(N % 2 == 0 && H >= 0 && 4 * H < N, "even length, alias-free window");
  constexpr int M = N / 2;
  C a[M];
  sfor<M>([&](auto nn) {
    constexpr int n = nn.value, i = n <= H ? n : n + M;
    if constexpr (in_win<M, H>(n)) a[n] = load(std::integral_constant<int, i>{});
    else a[n] = czero<C>();
  });
  if (par) {
    sfor<M>([&](auto nn) {
      constexpr int n = nn.value, i = n <= H ? n : n + M;
      if constexpr (in_win<M, H>(n)) a[n] = twmul<+1, i, N>(a[n]);
    });
  }
  line_fft<C, M, +1, H>([&](auto nn) { return a[nn.value]; }, store);
}

// Forward, the half of the inputs x[2n + par]: store(integral_constant<q>, v) with
// v = E[q] (par 0) or w_N^(-q) O[q] (par 1); X[k] = E[q] + O'[q] for k = q and
// E[q] - O'[q] for k = q + M.
template <typename C, int N, class L, class S>
__device__ __forceinline__ void half_forward(int par, L&& load, S&& store) {
  static_assert(N % 2 == 0, "even length");
  constexpr int M = N / 2;
  C o[M];
  line_fft<C, M, -1, -1>(load, [&](auto qq, C v) { o[qq.value] = v; });
  if (par) {
    sfor<M>([&](auto qq) { o[qq.value] = twmul<-1, qq.value, N>(o[qq.value]); });
  }
  sfor<M>([&](auto qq) { store(qq, o[qq.value]); });
}

}  // namespace ln
}  // namespace jrg
