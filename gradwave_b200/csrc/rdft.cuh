// Whole-transform DFTs in registers: one thread holds all N points of a
// transform in a local array and runs a fully unrolled mixed-radix
// decimation-in-time Cooley-Tukey recursion over it (N = R M: R interleaved
// M-point DFTs, twiddles W_N^(r k), R-point DFTs across them; Cooley & Tukey,
// Math. Comp. 19 (1965) 297; Van Loan, "Computational Frameworks for the
// FFT", 1992, sec. 2.3). The recursion works in place on strided views of the
// one array, every index and every twiddle is a compile-time constant, so the
// array lives in registers and a twiddle is an immediate operand; no shared
// memory, no barriers. Meant for the factors (up to 25 points) of the box axes
// that one thread holds.
//
// The twiddle constants cos/sin(2 pi k / N) come from a constexpr evaluator
// (quarter-turn reduction on the integer ratio k/N, then Taylor series on
// [-pi/4, pi/4] in sums of two doubles) and are rounded once.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace gwb {
namespace rdft_detail {

// Unevaluated sums h + l of two doubles, for the constants only (Dekker, Numer.
// Math. 18 (1971) 224).
struct dd {
  double h, l;
};
constexpr dd two_sum(double a, double b) {
  const double s = a + b, t = s - a;
  return {s, (a - (s - t)) + (b - t)};
}
constexpr dd two_prod(double a, double b) {
  const double ca = 134217729.0 * a, cb = 134217729.0 * b;
  const double ah = ca - (ca - a), al = a - ah, bh = cb - (cb - b), bl = b - bh;
  const double p = a * b;
  return {p, ((ah * bh - p) + ah * bl + al * bh) + al * bl};
}
constexpr dd add(dd a, dd b) {
  const dd s = two_sum(a.h, b.h);
  return two_sum(s.h, s.l + (a.l + b.l));
}
constexpr dd mul(dd a, dd b) {
  const dd p = two_prod(a.h, b.h);
  return two_sum(p.h, p.l + (a.h * b.l + a.l * b.h));
}
constexpr dd div(dd a, double d) {
  const double q = a.h / d;
  const dd p = two_prod(q, d);
  return two_sum(q, ((a.h - p.h) - p.l + a.l) / d);
}
// x - x^3/3! + ... (odd) or 1 - x^2/2! + ..., |x| <= pi/4
constexpr double sin_cos_series(dd x, bool odd) {
  const dd x2 = mul(x, x);
  dd term = odd ? x : dd{1.0, 0.0}, sum = term;
  for (int n = 1; n < 12; ++n) {
    term = div(mul(term, x2), -(odd ? 2.0 * n * (2.0 * n + 1.0) : (2.0 * n - 1.0) * (2.0 * n)));
    sum = add(sum, term);
  }
  return sum.h;
}
// cos(2 pi k / n) (which = 0) or sin(2 pi k / n) (which = 1), rounded to nearest:
// a constant off by a few units changes the length of what it rotates, and that
// error adds up in phase over the passes (density of a 49 x 50 x 14 box against
// extended precision: 5.7e-16 with constants good to a few units, 2.3e-16).
constexpr double cis(long k, long n, int which) {
  k %= n;
  if (k < 0) k += n;
  const long q = (8 * k + n) / (2 * n);  // nearest quarter turn
  const dd two_pi = {6.283185307179586, 2.4492935982947064e-16};
  const dd x = div(mul(two_pi, dd{(double)(4 * k - q * n), 0.0}), 4.0 * (double)n);
  const double c = sin_cos_series(x, false), s = sin_cos_series(x, true);
  switch (q % 4) {
    case 0: return which == 0 ? c : s;
    case 1: return which == 0 ? -s : c;
    case 2: return which == 0 ? -c : -s;
    default: return which == 0 ? s : -c;
  }
}

constexpr int first_radix(int n) {
  return n % 4 == 0 ? 4 : (n % 3 == 0 ? 3 : (n % 2 == 0 ? 2 : (n % 5 == 0 ? 5 : (n % 7 == 0 ? 7 : n))));
}

template <int I, int N>
struct StaticFor {
  template <class F>
  __host__ __device__ __forceinline__ static void run(F&& f) {
    if constexpr (I < N) {
      f(std::integral_constant<int, I>{});
      StaticFor<I + 1, N>::run(f);
    }
  }
};

// v * exp(SIGN 2 pi i K / N) with compile-time K, N
template <int N, int K, int SIGN, typename T>
__host__ __device__ __forceinline__ cplx<T> twiddle(cplx<T> v) {
  constexpr int k = ((K % N) + N) % N;
  if constexpr (k == 0) {
    return v;
  } else if constexpr (2 * k == N) {
    return mk<T>(-v.x, -v.y);
  } else if constexpr (4 * k == N) {
    return SIGN > 0 ? mk<T>(-v.y, v.x) : mk<T>(v.y, -v.x);
  } else if constexpr (4 * k == 3 * N) {
    return SIGN > 0 ? mk<T>(v.y, -v.x) : mk<T>(-v.y, v.x);
  } else {
    constexpr double cd = cis(k, N, 0), sd = SIGN * cis(k, N, 1);
    const T c = (T)cd, s = (T)sd;
    return mk<T>(v.x * c - v.y * s, v.x * s + v.y * c);
  }
}

template <int R, int SIGN, typename T>
__host__ __device__ __forceinline__ void small_dft(cplx<T> (&t)[R]) {
  if constexpr (R == 2) {
    const cplx<T> a = t[0], b = t[1];
    t[0] = a + b;
    t[1] = a - b;
  } else if constexpr (R == 3) {
    const T h = (T)0.86602540378443864676;
    const cplx<T> s1 = t[1] + t[2], d = t[1] - t[2];
    const cplx<T> m = mk<T>(t[0].x - (T)0.5 * s1.x, t[0].y - (T)0.5 * s1.y);
    // SIGN i sqrt3/2 d
    const cplx<T> q = SIGN > 0 ? mk<T>(-h * d.y, h * d.x) : mk<T>(h * d.y, -h * d.x);
    t[0] = t[0] + s1;
    t[1] = m + q;
    t[2] = m - q;
  } else if constexpr (R == 4) {
    const cplx<T> a0 = t[0] + t[2], a1 = t[0] - t[2];
    const cplx<T> b0 = t[1] + t[3], dd = t[1] - t[3];
    const cplx<T> b1 = SIGN > 0 ? mk<T>(-dd.y, dd.x) : mk<T>(dd.y, -dd.x);
    t[0] = a0 + b0;
    t[2] = a0 - b0;
    t[1] = a1 + b1;
    t[3] = a1 - b1;
  } else if constexpr (R == 6) {
    // coprime factors, no twiddles (Good, J. R. Stat. Soc. B 20 (1958) 361):
    // input 3 a + 2 b, output 3 k + 4 l (mod 6). As 3 x 2 with twiddles the
    // rounding of sin(pi / 3) enters twice per pass, always with one sign.
    cplx<T> u[3] = {t[0], t[2], t[4]}, v[3] = {t[3], t[5], t[1]};
    small_dft<3, SIGN>(u);
    small_dft<3, SIGN>(v);
    t[0] = u[0] + v[0], t[3] = u[0] - v[0];
    t[4] = u[1] + v[1], t[1] = u[1] - v[1];
    t[2] = u[2] + v[2], t[5] = u[2] - v[2];
  } else if constexpr (R == 5 || R == 7) {
    // odd prime length: with s_j = t_j + t_(R-j), d_j = t_j - t_(R-j),
    // X_k = t_0 + sum_j cos(2 pi j k / R) s_j + SIGN i sum_j sin(2 pi j k / R) d_j
    // and X_(R-k) the same with the second sum subtracted
    constexpr int H = (R - 1) / 2;
    cplx<T> s[H], d[H];
    const cplx<T> t0 = t[0];
    cplx<T> sum = t0;
    StaticFor<0, H>::run([&](auto jc) {
      constexpr int j = decltype(jc)::value;
      s[j] = t[j + 1] + t[R - 1 - j];
      d[j] = t[j + 1] - t[R - 1 - j];
      sum = sum + s[j];
    });
    t[0] = sum;
    StaticFor<0, H>::run([&](auto kc) {
      constexpr int k = decltype(kc)::value + 1;
      cplx<T> a = t0, b = mk<T>((T)0, (T)0);
      StaticFor<0, H>::run([&](auto jc) {
        constexpr int j = decltype(jc)::value;
        constexpr double cd = cis((long)(j + 1) * k, R, 0), sd = SIGN * cis((long)(j + 1) * k, R, 1);
        a = mk<T>(a.x + (T)cd * s[j].x, a.y + (T)cd * s[j].y);
        b = mk<T>(b.x + (T)sd * d[j].x, b.y + (T)sd * d[j].y);
      });
      t[k] = mk<T>(a.x - b.y, a.y + b.x);
      t[R - k] = mk<T>(a.x + b.y, a.y - b.x);
    });
  }
}

// Position, within a length-N subsequence, where the in-place recursion below
// leaves output X[k]: for N = R M, X[kk + M q] lands where sub-DFT q kept its
// output kk, i.e. at q + R pos_M(kk) (digit reversal over the radix chain).
constexpr int out_pos(int n, int k) {
  if (n <= 7) return k;
  const int r = first_radix(n), m = n / r;
  return (k / m) + r * out_pos(m, k % m);
}

// In-place DFT of the length-N subsequence x[OFF + STRIDE i], outputs in
// out_pos order.
template <int N, int SIGN, int OFF, int STRIDE, typename T, int NT>
__host__ __device__ __forceinline__ void dit_ip(cplx<T> (&x)[NT]) {
  if constexpr (N == 1) {
    return;
  } else if constexpr (N <= 7) {
    cplx<T> t[N];
    StaticFor<0, N>::run([&](auto ic) { t[decltype(ic)::value] = x[OFF + STRIDE * decltype(ic)::value]; });
    small_dft<N, SIGN>(t);
    StaticFor<0, N>::run([&](auto ic) { x[OFF + STRIDE * decltype(ic)::value] = t[decltype(ic)::value]; });
  } else {
    constexpr int R = first_radix(N);
    constexpr int M = N / R;
    static_assert(R * M == N && R <= 7, "rdft: lengths with prime factors 2, 3, 5 and 7 only");
    StaticFor<0, R>::run([&](auto rc) {
      constexpr int r = decltype(rc)::value;
      dit_ip<M, SIGN, OFF + STRIDE * r, STRIDE * R>(x);
    });
    StaticFor<0, M>::run([&](auto kc) {
      constexpr int kk = decltype(kc)::value;
      constexpr int slot = STRIDE * R * out_pos(M, kk);  // where every sub-DFT keeps its output kk
      cplx<T> t[R];
      StaticFor<0, R>::run([&](auto rc) {
        constexpr int r = decltype(rc)::value;
        t[r] = twiddle<N, r * kk, SIGN>(x[OFF + STRIDE * r + slot]);
      });
      small_dft<R, SIGN>(t);
      StaticFor<0, R>::run([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        x[OFF + STRIDE * q + slot] = t[q];
      });
    });
  }
}

}  // namespace rdft_detail

// DFT of x (natural order): X[k] = sum_n x[n] exp(SIGN 2 pi i n k / N),
// unnormalised, left in x at position out_pos(N, k).
template <int N, int SIGN, typename T>
__host__ __device__ __forceinline__ void rdft_perm(cplx<T> (&x)[N]) {
  rdft_detail::dit_ip<N, SIGN, 0, 1>(x);
}

// The same with the output in natural order (a compile-time renaming).
template <int N, int SIGN, typename T>
__host__ __device__ __forceinline__ void rdft(cplx<T> (&x)[N]) {
  using namespace rdft_detail;
  rdft_perm<N, SIGN>(x);
  cplx<T> y[N];
  StaticFor<0, N>::run([&](auto kc) {
    constexpr int k = decltype(kc)::value;
    y[k] = x[out_pos(N, k)];
  });
  StaticFor<0, N>::run([&](auto kc) { x[decltype(kc)::value] = y[decltype(kc)::value]; });
}

}  // namespace gwb
