// One-axis FFT kernels of the local term, for every box axis length 2^a 3^b
// 5^c 7^d <= 128 (the 52 lengths of GWB_FFT_LENGTHS, one instantiation each).
//
// A length N is split as N = R1 R2 (both <= 16; 125 = 5 x 25; lengths up to 16
// are not split). With n = a + R2 b and k = k1 + R1 k2,
//
//   X[k1 + R1 k2] = sum_a w_R2^(a k2) [ w_N^(a k1) sum_b w_R1^(b k1) x[a + R2 b] ]
//
// so a thread that holds the R1 points x[a + R2 b] transforms them in registers
// (rdft.cuh), multiplies by the twiddles w_N^(a k1) and hands them through
// shared memory to the thread that holds the R2 points of one k1 (Cooley &
// Tukey, Math. Comp. 19 (1965) 297). Two register passes and one exchange per
// axis: a pass per radix in shared memory, as these kernels had it before, cost
// three to four exchanges with two block barriers each, and a block that holds a
// whole plane leaves room for one to three blocks per SM.
//
// Kernels (k = k-point, b = band of the chunk):
//   k_rows_inverse   sphere -> W2: axis 2 of the occupied rows (j0, i1); the
//                    coefficients go from c straight to registers (map)
//   k_cols_inverse   W2 -> W: axis 1 of the occupied planes j0, all n2 columns
//   k_pencil_vloc    W -> W: axis 0, times v(r)/N, axis 0 back
//   k_cols_forward   W -> W2: axis 1, the occupied rows only
//   k_rows_forward   W2 -> out: axis 2, gathered to the sphere, + t c
//   k_pencil_density W -> rho: axis 0 and sum of w |psi|^2 over a band group
// Rows and columns are separate launches so that each kernel needs only its own
// axis length and a few tens of KB of shared memory; the price is W2 (the rows
// of the sphere's disc, 0.4 of W) written and read once more each way. Measured
// against the passes in shared memory (whole applies, us; in brackets with the
// predicates, twiddle layout and prefetch below, chained launches and the
// products of zmma.cuh): 42^3 float32 240 rows 1086 -> 212 (181), 36x36x108
// float64 244 rows 2760 -> 763 (585), 84^3 float64 258 rows 13836 -> 5513 (3733),
// 108^3 float32 166 rows 14936 -> 3096 (2678), 96^3 float64 240 rows 12031 -> 7830
// (7505). Bound by issue and the float64 pipe in the pencils, by latency in the
// others (up to 4 TB/s of scratch traffic), not by HBM.
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"
#include "rdft.cuh"

namespace gwb {

#define GWB_FFT_LENGTHS(X)                                                                                     \
  X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(12) X(14) X(15) X(16) X(18) X(20) X(21) X(24) X(25) X(27)    \
  X(28) X(30) X(32) X(35) X(36) X(40) X(42) X(45) X(48) X(49) X(50) X(54) X(56) X(60) X(63) X(64) X(70) X(72)  \
  X(75) X(80) X(81) X(84) X(90) X(96) X(98) X(100) X(105) X(108) X(112) X(120) X(125) X(126) X(128)

// What one chunk of bands of the local term (or the density) works on.
template <typename T> struct FftRun {
  int n0, n1, n2;        // box
  int M0, L0, M2;        // occupied extents of axes 0 and 2 (M = n: all of the axis)
  int nk, nrow;          // k-points, row slots per k of W2
  int nbc, b0;           // bands of this chunk, first band
  int npw_max;
  const int* map;        // (nk, nrow, n2) sphere index of each row point, -1: none
  const int* rowof;      // (nk, L0, n1) row slot of (j0, i1), -1: none
  const int* npw;        // (nk)
  const cplx<T>* tw0;    // per axis, n = R1 R2: exp(-2 pi i a k / n) at k R2 + a, a < R2, k < R1
  const cplx<T>* tw1;
  const cplx<T>* tw2;
  cplx<T>* W2;           // (nk, nbc, nrow, n2)
  cplx<T>* W;            // (nk, nbc, L0, n1, n2)
  const T* v;            // (n0, n1, n2) v(r) / N
  const T* t;            // (nk, npw_max)
  const void* c;         // rows (nk, ., npw_max), complex128 when io64 else complex64
  void* out;
  int64_t ck, ok;        // k strides of c and out
  int io64;
  // density
  const double* w;       // (nk, .) band weights, k stride wk
  int64_t wk;
  double* rho;           // (nk, ngrp, n0, n1, n2)
  int ngrp, first;       // band groups; first: start from zero
};

// R1 of N = R1 R2, R1 <= R2 (R2 = 1: not split)
constexpr int fft_r1(int n) {
  if (n <= 16) return n;
  int best = 0;
  for (int r = 2; r * r <= n; ++r)
    if (n % r == 0 && (n / r <= 16 || n == 125)) best = r;
  return best;
}

template <typename T, int N> struct AxisCfg {
  static constexpr int R1 = fft_r1(N), R2 = N / R1;
  static_assert(R1 * R2 == N && R1 > 0, "axis length without a split");
  // strided pencils per block (consecutive lanes take consecutive pencils, so a
  // warp's loads are whole 128-byte lines); two passes: R2 threads per pencil
  static constexpr int PB = R2 == 1 ? 128 : (R2 >= 8 ? 16 : 32);
  static constexpr int NT = PB * R2;
  // contiguous rows per block; padded so that a column of the exchange (one
  // element per row of R2) hits different banks
  static constexpr int P2 = R2 | 1;
  static constexpr int RB = R2 == 1 ? 64 : (192 / R2 > 0 ? 192 / R2 : 1);
  static constexpr int NTR = RB * R2;
  // blocks per SM the registers are limited for (at most 113 registers in
  // float64, 64 in float32; the 25-point pass of 125 needs more)
  static constexpr int minb(int nt, int threads = sizeof(T) == 8 ? 576 : 1024) {
    const int t = R2 == 1 ? threads * 5 / 8 : threads;  // one pass holds all N points
    return R2 > 16 || t < nt ? 1 : t / nt;
  }
  static constexpr size_t smem_strided = R2 == 1 ? 0 : (size_t)N * PB * sizeof(cplx<T>);
  static constexpr size_t smem_rows = R2 == 1 ? 0 : (size_t)RB * R1 * P2 * sizeof(cplx<T>);
};

namespace fft_detail {

using rdft_detail::StaticFor;

template <int SIGN, typename T> __device__ __forceinline__ cplx<T> tw_at(const cplx<T>* tw) {
  const cplx<T> w = *tw;
  return SIGN > 0 ? conj(w) : w;
}

// First pass: R1 points x[a + R2 b] -> exchange slots [k1][a], twiddled; twa =
// the axis table at column a (row k1: w_N^(a k1)), so that every twiddle is a
// load at a constant offset.
template <typename T, int R1, int R2, int SIGN, class PUT>
__device__ __forceinline__ void pass1(cplx<T> (&x)[R1], const cplx<T>* __restrict__ twa, PUT&& put) {
  rdft<R1, SIGN>(x);
  StaticFor<0, R1>::run([&](auto kc) {
    constexpr int k1 = decltype(kc)::value;
    put(k1, k1 == 0 ? x[0] : x[k1] * tw_at<SIGN>(twa + k1 * R2));
  });
}

// Loads (0 where p is false) and stores under a predicate: written as branches
// they took 40 % of the branch unit's cycles and a third of the issue slots of
// the float32 kernels.
__device__ __forceinline__ cplx<double> ld_if(bool p, const cplx<double>* a) {
  cplx<double> v;
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %3, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t"
      "mov.f64 %1, 0d0000000000000000;\n\t@q ld.global.v2.f64 {%0, %1}, [%2];\n\t}"
      : "=&d"(v.x), "=&d"(v.y)
      : "l"(a), "r"((int)p)
      : "memory");
  return v;
}
__device__ __forceinline__ cplx<float> ld_if(bool p, const cplx<float>* a) {
  cplx<float> v;
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %3, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
      "mov.f32 %1, 0f00000000;\n\t@q ld.global.v2.f32 {%0, %1}, [%2];\n\t}"
      : "=&f"(v.x), "=&f"(v.y)
      : "l"(a), "r"((int)p)
      : "memory");
  return v;
}
__device__ __forceinline__ void st_if(bool p, cplx<double>* a, cplx<double> v) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %3, 0;\n\t@q st.global.v2.f64 [%0], {%1, %2};\n\t}" ::"l"(a),
               "d"(v.x), "d"(v.y), "r"((int)p)
               : "memory");
}
__device__ __forceinline__ void st_if(bool p, cplx<float>* a, cplx<float> v) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %3, 0;\n\t@q st.global.v2.f32 [%0], {%1, %2};\n\t}" ::"l"(a),
               "f"(v.x), "f"(v.y), "r"((int)p)
               : "memory");
}

// element i of a complex128 or complex64 array (0 where i < 0) in precision T
template <typename T, typename SIO> __device__ __forceinline__ cplx<T> load_io(const SIO* p, int i) {
  const SIO v = ld_if(i >= 0, p + i);
  return mk<T>((T)v.x, (T)v.y);
}

// one complex element, global to shared memory, asynchronously (0 where p is false)
template <typename T> __device__ __forceinline__ void cp_async_elem(bool p, cplx<T>* dst, const cplx<T>* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = p ? (int)sizeof(cplx<T>) : 0;
  if constexpr (sizeof(cplx<T>) == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

// memory row r of axis 0 -> offset of its occupied plane in W, or -1
__device__ __forceinline__ int plane_of(int r, int M0, int L0, int n0, int plane) {
  if (r <= M0) return r * plane;
  return r >= n0 - (L0 - M0 - 1) ? (r - (n0 - L0)) * plane : -1;
}

}  // namespace fft_detail

template <typename T, int N>
__global__ void __launch_bounds__(AxisCfg<T, N>::NTR, AxisCfg<T, N>::minb(AxisCfg<T, N>::NTR))
    k_rows_inverse(const FftRun<T> f) {
  using C = AxisCfg<T, N>;
  using namespace fft_detail;
  constexpr int R1 = C::R1, R2 = C::R2, P2 = C::P2, RB = C::RB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* ex = reinterpret_cast<cplx<T>*>(smem_raw);
  const int bl = blockIdx.y, k = blockIdx.z, tid = threadIdx.x;
  const int row0 = blockIdx.x * RB;
  const size_t crow = (size_t)k * f.ck + (size_t)(f.b0 + bl) * f.npw_max;
  {
    const int a = tid % R2, r = tid / R2, row = row0 + r;
    if (row < f.nrow) {
      const int* mp = f.map + ((size_t)k * f.nrow + row) * N;
      int idx[R1];
      StaticFor<0, R1>::run([&](auto bc) {
        constexpr int b = decltype(bc)::value;
        const int i2 = a + R2 * b;
        idx[b] = (i2 <= f.M2 || i2 >= N - f.M2) ? mp[i2] : -1;
      });
      chain_wait();
      cplx<T> x[R1];
      if (f.io64) {
        const cplx<double>* c = (const cplx<double>*)f.c + crow;
        StaticFor<0, R1>::run([&](auto bc) { x[decltype(bc)::value] = load_io<T>(c, idx[decltype(bc)::value]); });
      } else {
        const cplx<float>* c = (const cplx<float>*)f.c + crow;
        StaticFor<0, R1>::run([&](auto bc) { x[decltype(bc)::value] = load_io<T>(c, idx[decltype(bc)::value]); });
      }
      if constexpr (R2 == 1) {
        rdft<R1, +1>(x);
        cplx<T>* dst = f.W2 + (((size_t)k * f.nbc + bl) * f.nrow + row) * N;
        StaticFor<0, R1>::run([&](auto bc) { dst[decltype(bc)::value] = x[decltype(bc)::value]; });
      } else {
        cplx<T>* e = ex + r * (R1 * P2) + a;
        pass1<T, R1, R2, +1>(x, f.tw2 + a, [&](int k1, cplx<T> v) { e[k1 * P2] = v; });
      }
    }
  }
  if constexpr (R2 > 1) {
    __syncthreads();
    const int k1 = tid % R1, r = tid / R1, row = row0 + r;
    if (r < RB && row < f.nrow) {
      const cplx<T>* e = ex + r * (R1 * P2) + k1 * P2;
      cplx<T> y[R2];
      StaticFor<0, R2>::run([&](auto ac) { y[decltype(ac)::value] = e[decltype(ac)::value]; });
      rdft<R2, +1>(y);
      cplx<T>* dst = f.W2 + (((size_t)k * f.nbc + bl) * f.nrow + row) * N + k1;
      StaticFor<0, R2>::run([&](auto kc) { dst[R1 * decltype(kc)::value] = y[decltype(kc)::value]; });
    }
  }
}

template <typename T, int N>
__global__ void __launch_bounds__(AxisCfg<T, N>::NTR, AxisCfg<T, N>::minb(AxisCfg<T, N>::NTR))
    k_rows_forward(const FftRun<T> f) {
  using C = AxisCfg<T, N>;
  using namespace fft_detail;
  constexpr int R1 = C::R1, R2 = C::R2, P2 = C::P2, RB = C::RB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* ex = reinterpret_cast<cplx<T>*>(smem_raw);
  const int bl = blockIdx.y, k = blockIdx.z, tid = threadIdx.x;
  const int row0 = blockIdx.x * RB;
  const size_t crow = (size_t)k * f.ck + (size_t)(f.b0 + bl) * f.npw_max;
  const size_t orow = (size_t)k * f.ok + (size_t)(f.b0 + bl) * f.npw_max;
  const T* tk = f.t + (size_t)k * f.npw_max;
  chain_wait();
  auto store = [&](int g, cplx<T> val) {  // where g >= 0
    const T tg = g >= 0 ? tk[g] : (T)0;
    if (f.io64) {
      const cplx<T> o = val + scale(load_io<T>((const cplx<double>*)f.c + crow, g), tg);
      st_if(g >= 0, (cplx<double>*)f.out + orow + g, mk<double>(o.x, o.y));
    } else {
      const cplx<T> o = val + scale(load_io<T>((const cplx<float>*)f.c + crow, g), tg);
      st_if(g >= 0, (cplx<float>*)f.out + orow + g, mk<float>((float)o.x, (float)o.y));
    }
  };
  {
    const int a = tid % R2, r = tid / R2, row = row0 + r;
    if (row < f.nrow) {
      const cplx<T>* src = f.W2 + (((size_t)k * f.nbc + bl) * f.nrow + row) * N + a;
      cplx<T> x[R1];
      StaticFor<0, R1>::run([&](auto bc) { x[decltype(bc)::value] = src[R2 * decltype(bc)::value]; });
      if constexpr (R2 == 1) {
        rdft<R1, -1>(x);
        const int* mp = f.map + ((size_t)k * f.nrow + row) * N;
        StaticFor<0, R1>::run([&](auto bc) {
          store(mp[decltype(bc)::value], x[decltype(bc)::value]);
        });
      } else {
        cplx<T>* e = ex + r * (R1 * P2) + a;
        pass1<T, R1, R2, -1>(x, f.tw2 + a, [&](int k1, cplx<T> v) { e[k1 * P2] = v; });
      }
    }
  }
  if constexpr (R2 > 1) {
    __syncthreads();
    const int k1 = tid % R1, r = tid / R1, row = row0 + r;
    if (r < RB && row < f.nrow) {
      const int* mp = f.map + ((size_t)k * f.nrow + row) * N + k1;
      const cplx<T>* e = ex + r * (R1 * P2) + k1 * P2;
      cplx<T> y[R2];
      StaticFor<0, R2>::run([&](auto ac) { y[decltype(ac)::value] = e[decltype(ac)::value]; });
      rdft<R2, -1>(y);
      StaticFor<0, R2>::run([&](auto kc) {
        constexpr int o = R1 * decltype(kc)::value;
        const int i2 = k1 + o;
        const int g = (i2 <= f.M2 || i2 >= N - f.M2) ? mp[o] : -1;
        store(g, y[decltype(kc)::value]);
      });
    }
  }
  if (blockIdx.x == 0) {
    for (int g = f.npw[k] + tid; g < f.npw_max; g += blockDim.x) {
      if (f.io64) st((cplx<double>*)f.out, orow + g, mk<T>(0, 0));
      else st((cplx<float>*)f.out, orow + g, mk<T>(0, 0));
    }
  }
}

// Axis 1 of the columns (j0, i2) of one (band, k); columns are numbered
// q = j0 n2 + i2, so that neighbouring lanes take neighbouring i2.
template <typename T, int N>
__global__ void __launch_bounds__(AxisCfg<T, N>::NT, AxisCfg<T, N>::minb(AxisCfg<T, N>::NT))
    k_cols_inverse(const FftRun<T> f) {
  using C = AxisCfg<T, N>;
  using namespace fft_detail;
  constexpr int R1 = C::R1, R2 = C::R2, PB = C::PB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* ex = reinterpret_cast<cplx<T>*>(smem_raw);
  const int bl = blockIdx.y, k = blockIdx.z, n2 = f.n2;
  const int c = threadIdx.x % PB, s = threadIdx.x / PB;
  const int q = blockIdx.x * PB + c;
  const bool live = q < f.L0 * n2;
  const int j0 = live ? q / n2 : 0, i2 = q - j0 * n2;
  const size_t kb = (size_t)k * f.nbc + bl;
  if (live) {
    const int* ro = f.rowof + ((size_t)k * f.L0 + j0) * N + s;
    const cplx<T>* src = f.W2 + kb * f.nrow * n2 + i2;
    int idx[R1];
    StaticFor<0, R1>::run([&](auto bc) { idx[decltype(bc)::value] = ro[R2 * decltype(bc)::value]; });
    chain_wait();
    cplx<T> x[R1];
    StaticFor<0, R1>::run([&](auto bc) {
      constexpr int b = decltype(bc)::value;
      x[b] = ld_if(idx[b] >= 0, src + idx[b] * n2);
    });
    if constexpr (R2 == 1) {
      rdft<R1, +1>(x);
      cplx<T>* dst = f.W + (kb * f.L0 + j0) * (size_t)(N * n2) + i2;
      StaticFor<0, R1>::run([&](auto bc) { dst[decltype(bc)::value * n2] = x[decltype(bc)::value]; });
    } else {
      cplx<T>* e = ex + s * PB + c;
      pass1<T, R1, R2, +1>(x, f.tw1 + s, [&](int k1, cplx<T> v) { e[k1 * (R2 * PB)] = v; });
    }
  }
  if constexpr (R2 > 1) {
    __syncthreads();
    if (s < R1 && live) {
      const cplx<T>* e = ex + s * (R2 * PB) + c;
      cplx<T> y[R2];
      StaticFor<0, R2>::run([&](auto ac) { y[decltype(ac)::value] = e[decltype(ac)::value * PB]; });
      rdft<R2, +1>(y);
      cplx<T>* dst = f.W + (kb * f.L0 + j0) * (size_t)(N * n2) + (size_t)s * n2 + i2;
      StaticFor<0, R2>::run([&](auto kc) { dst[R1 * decltype(kc)::value * n2] = y[decltype(kc)::value]; });
    }
  }
}

template <typename T, int N>
__global__ void __launch_bounds__(AxisCfg<T, N>::NT, AxisCfg<T, N>::minb(AxisCfg<T, N>::NT))
    k_cols_forward(const FftRun<T> f) {
  using C = AxisCfg<T, N>;
  using namespace fft_detail;
  constexpr int R1 = C::R1, R2 = C::R2, PB = C::PB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* ex = reinterpret_cast<cplx<T>*>(smem_raw);
  const int bl = blockIdx.y, k = blockIdx.z, n2 = f.n2;
  const int c = threadIdx.x % PB, s = threadIdx.x / PB;
  const int q = blockIdx.x * PB + c;
  const bool live = q < f.L0 * n2;
  const int j0 = live ? q / n2 : 0, i2 = q - j0 * n2;
  const size_t kb = (size_t)k * f.nbc + bl;
  cplx<T>* dst = f.W2 + kb * f.nrow * n2 + i2;
  const int* ro = f.rowof + ((size_t)k * f.L0 + j0) * N;
  chain_wait();
  if (live) {
    const cplx<T>* src = f.W + (kb * f.L0 + j0) * (size_t)(N * n2) + (size_t)s * n2 + i2;
    cplx<T> x[R1];
    StaticFor<0, R1>::run([&](auto bc) { x[decltype(bc)::value] = src[R2 * decltype(bc)::value * n2]; });
    if constexpr (R2 == 1) {
      rdft<R1, -1>(x);
      StaticFor<0, R1>::run([&](auto bc) {
        const int row = ro[decltype(bc)::value];
        st_if(row >= 0, dst + row * n2, x[decltype(bc)::value]);
      });
    } else {
      cplx<T>* e = ex + s * PB + c;
      pass1<T, R1, R2, -1>(x, f.tw1 + s, [&](int k1, cplx<T> v) { e[k1 * (R2 * PB)] = v; });
    }
  }
  if constexpr (R2 > 1) {
    __syncthreads();
    if (s < R1 && live) {
      const cplx<T>* e = ex + s * (R2 * PB) + c;
      cplx<T> y[R2];
      StaticFor<0, R2>::run([&](auto ac) { y[decltype(ac)::value] = e[decltype(ac)::value * PB]; });
      rdft<R2, -1>(y);
      StaticFor<0, R2>::run([&](auto kc) {
        constexpr int k2 = decltype(kc)::value;
        const int row = ro[s + R1 * k2];
        st_if(row >= 0, dst + row * n2, y[k2]);
      });
    }
  }
}

// Axis 0 of the pencils p = i1 n2 + i2 of a group of bands: inverse, times
// v(r)/N, forward. After the inverse a thread holds the R2 points
// i0 = k1 + R1 k2 of its pencil; the forward transform starts on exactly these
// (DFT over k2 first, twiddle w_N^(k1 m2), exchange, DFT over k1), so the pair
// costs two exchanges, in place in one buffer. v is read from L1 after the
// first band of the group (kept in registers it made the float64 kernels
// spill). The next band's points travel to shared memory while this band is
// transformed.
template <typename T, int N>
__global__ void __launch_bounds__(AxisCfg<T, N>::NT, AxisCfg<T, N>::minb(AxisCfg<T, N>::NT))
    k_pencil_vloc(const FftRun<T> f, int bands_per_block) {
  using C = AxisCfg<T, N>;
  using namespace fft_detail;
  constexpr int R1 = C::R1, R2 = C::R2, PB = C::PB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* ex = reinterpret_cast<cplx<T>*>(smem_raw);
  cplx<T>* in = ex + N * PB + threadIdx.x;  // this thread's R1 points of the next band, NT apart
  const int k = blockIdx.z;
  const int plane = f.n1 * f.n2;  // box indices fit 32 bits (axes <= 128)
  const int c = threadIdx.x % PB, s = threadIdx.x / PB;
  const int p = blockIdx.x * PB + c;
  const bool live = p < plane;
  const int M0 = f.M0, L0 = f.L0;
  const int bl0 = blockIdx.y * bands_per_block, bl1 = min(f.nbc, bl0 + bands_per_block);
  int off[R1];  // planes of the pencil's points s + R2 b in W
  StaticFor<0, R1>::run([&](auto bc) {
    constexpr int b = decltype(bc)::value;
    off[b] = plane_of(s + R2 * b, M0, L0, N, plane);
  });
  auto band = [&](int bl) { return f.W + ((size_t)k * f.nbc + bl) * (size_t)(L0 * plane) + p; };
  auto fetch = [&](int bl) {
    if (live && bl < bl1) {
      const cplx<T>* base = band(bl);
      StaticFor<0, R1>::run([&](auto bc) {
        constexpr int b = decltype(bc)::value;
        cp_async_elem(off[b] >= 0, in + b * C::NT, base + max(off[b], 0));
      });
    }
    cp_async_commit();
  };
  chain_wait();
  if constexpr (R2 > 1) fetch(bl0);
  for (int bl = bl0; bl < bl1; ++bl) {
    // opaque per band: hoisted out of the loop, the twiddles and the addresses
    // take more registers than there are
    const T* vp = f.v + p + s * plane;
    const cplx<T>* tw = f.tw0;
    asm volatile("" : "+l"(vp), "+l"(tw));
    cplx<T>* base = band(bl);
    if constexpr (R2 == 1) {
      if (live) {
        cplx<T> x[R1];
        StaticFor<0, R1>::run([&](auto bc) {
          constexpr int b = decltype(bc)::value;
          x[b] = ld_if(off[b] >= 0, base + off[b]);
        });
        rdft<R1, +1>(x);
        StaticFor<0, R1>::run([&](auto bc) {
          x[decltype(bc)::value] = scale(x[decltype(bc)::value], vp[decltype(bc)::value * plane]);
        });
        rdft<R1, -1>(x);
        StaticFor<0, R1>::run([&](auto bc) {
          constexpr int b = decltype(bc)::value;
          st_if(off[b] >= 0, base + off[b], x[b]);
        });
      }
    } else {
      cp_async_wait<0>();  // the points are this thread's own: no barrier
      if (live) {
        cplx<T> x[R1];
        StaticFor<0, R1>::run([&](auto bc) {
          constexpr int b = decltype(bc)::value;
          x[b] = in[b * C::NT];
        });
        cplx<T>* e = ex + s * PB + c;
        pass1<T, R1, R2, +1>(x, tw + s, [&](int k1, cplx<T> v) { e[k1 * (R2 * PB)] = v; });
      }
      fetch(bl + 1);
      __syncthreads();
      // the R2 points of one k1 are read and written by one thread: in place
      if (s < R1 && live) {
        cplx<T>* e = ex + s * (R2 * PB) + c;
        cplx<T> y[R2];
        StaticFor<0, R2>::run([&](auto ac) { y[decltype(ac)::value] = e[decltype(ac)::value * PB]; });
        rdft<R2, +1>(y);
        StaticFor<0, R2>::run([&](auto kc) {
          y[decltype(kc)::value] = scale(y[decltype(kc)::value], vp[R1 * decltype(kc)::value * plane]);
        });
        rdft<R2, -1>(y);
        StaticFor<0, R2>::run([&](auto mc) {
          constexpr int m2 = decltype(mc)::value;
          e[m2 * PB] = m2 == 0 ? y[0] : y[m2] * tw_at<-1>(tw + s * R2 + m2);
        });
      }
      __syncthreads();
      // column s of the exchange is read here and written by the next band's
      // first pass, both by this thread
      if (live) {
        const cplx<T>* e = ex + s * PB + c;
        cplx<T> x[R1];
        StaticFor<0, R1>::run([&](auto kc) { x[decltype(kc)::value] = e[decltype(kc)::value * (R2 * PB)]; });
        rdft<R1, -1>(x);
        StaticFor<0, R1>::run([&](auto bc) {
          constexpr int b = decltype(bc)::value;
          st_if(off[b] >= 0, base + off[b], x[b]);
        });
      }
    }
  }
}

// Density (gradwave core/batch.py:562-587, density_b): axis 0 of each pencil
// and rho[k][group][r] += w[k][b] |psi_b(r)|^2 over the chunk's bands of the
// group, in registers: one thread owns each output element, so the sums run in
// a fixed order without atomics.
template <typename T, int N>
__global__ void __launch_bounds__(AxisCfg<T, N>::NT, AxisCfg<T, N>::minb(AxisCfg<T, N>::NT, 448))
    k_pencil_density(const FftRun<T> f) {
  using C = AxisCfg<T, N>;
  using namespace fft_detail;
  constexpr int R1 = C::R1, R2 = C::R2, PB = C::PB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* ex1 = reinterpret_cast<cplx<T>*>(smem_raw);
  const int k = blockIdx.z, grp = blockIdx.y;
  const int plane = f.n1 * f.n2;  // box indices fit 32 bits (axes <= 128)
  const int c = threadIdx.x % PB, s = threadIdx.x / PB;
  const int p = blockIdx.x * PB + c;
  const bool live = p < plane;
  const int M0 = f.M0, L0 = f.L0;
  constexpr int RV = R2 == 1 ? R1 : R2, SV = R2 == 1 ? 1 : R1;
  const bool own = live && s < SV;
  double* rk = f.rho + ((size_t)k * f.ngrp + grp) * N * plane + p + (R2 == 1 ? 0 : s * plane);
  double acc[RV];
  chain_wait();
  StaticFor<0, RV>::run([&](auto kc) {
    acc[decltype(kc)::value] = own && !f.first ? rk[SV * decltype(kc)::value * plane] : 0.0;
  });
  int buf = 0;
  // band b belongs to group b % ngrp whatever the chunks are
  for (int bl = (grp + f.ngrp - f.b0 % f.ngrp) % f.ngrp; bl < f.nbc; bl += f.ngrp) {
    const double wb = f.w[(size_t)k * f.wk + f.b0 + bl];
    if (wb == 0.0) continue;  // the same for every thread of the block
    const cplx<T>* base = f.W + ((size_t)k * f.nbc + bl) * (size_t)(L0 * plane) + p;
    auto add = [&](double& a, cplx<T> z) { a += wb * ((double)z.x * (double)z.x + (double)z.y * (double)z.y); };
    cplx<T>* exb = ex1 + buf * (N * PB);
    const cplx<T>* tw = f.tw0;  // opaque per band, as in k_pencil_vloc
    int s_ = s;
    asm volatile("" : "+l"(tw), "+r"(s_));
    if (live) {
      cplx<T> x[R1];
      StaticFor<0, R1>::run([&](auto bc) {
        constexpr int b = decltype(bc)::value;
        const int o = plane_of(s_ + R2 * b, M0, L0, N, plane);
        x[b] = ld_if(o >= 0, base + o);
      });
      if constexpr (R2 == 1) {
        rdft<R1, +1>(x);
        StaticFor<0, R1>::run([&](auto bc) { add(acc[decltype(bc)::value], x[decltype(bc)::value]); });
      } else {
        cplx<T>* e = exb + s * PB + c;
        pass1<T, R1, R2, +1>(x, tw + s, [&](int k1, cplx<T> v) { e[k1 * (R2 * PB)] = v; });
      }
    }
    if constexpr (R2 > 1) {
      __syncthreads();  // the other buffer is free: its readers have arrived here too
      if (own) {
        const cplx<T>* e = exb + s * (R2 * PB) + c;
        cplx<T> y[R2];
        StaticFor<0, R2>::run([&](auto ac) { y[decltype(ac)::value] = e[decltype(ac)::value * PB]; });
        rdft<R2, +1>(y);
        StaticFor<0, R2>::run([&](auto kc) { add(acc[decltype(kc)::value], y[decltype(kc)::value]); });
      }
      buf ^= 1;
    }
  }
  if (own)
    StaticFor<0, RV>::run([&](auto kc) { rk[SV * decltype(kc)::value * plane] = acc[decltype(kc)::value]; });
}

// Launchers: cudaErrorInvalidValue when the axis length is not one of GWB_FFT_LENGTHS.
template <typename T> cudaError_t fft_rows_inverse(const FftRun<T>& f, cudaStream_t st);
template <typename T> cudaError_t fft_rows_forward(const FftRun<T>& f, cudaStream_t st);
template <typename T> cudaError_t fft_cols_inverse(const FftRun<T>& f, cudaStream_t st);
template <typename T> cudaError_t fft_cols_forward(const FftRun<T>& f, cudaStream_t st);
template <typename T> cudaError_t fft_pencil_vloc(const FftRun<T>& f, cudaStream_t st);
cudaError_t fft_pencil_density(const FftRun<double>& f, cudaStream_t st);

namespace fft_detail {

template <typename T, int N> cudaError_t launch_rows(void (*kern)(FftRun<T>), const FftRun<T>& f, cudaStream_t st) {
  using C = AxisCfg<T, N>;
  dim3 g((f.nrow + C::RB - 1) / C::RB, f.nbc, f.nk);
  return launch_chained(kern, g, C::NTR, C::smem_rows, st, f);
}

template <typename T, int N> cudaError_t launch_cols(void (*kern)(FftRun<T>), const FftRun<T>& f, cudaStream_t st) {
  using C = AxisCfg<T, N>;
  dim3 g((f.L0 * f.n2 + C::PB - 1) / C::PB, f.nbc, f.nk);
  return launch_chained(kern, g, C::NT, C::smem_strided, st, f);
}

template <typename T, int N> cudaError_t launch_vloc(const FftRun<T>& f, cudaStream_t st) {
  using C = AxisCfg<T, N>;
  const int blocks = (f.n1 * f.n2 + C::PB - 1) / C::PB;
  // bands per block: v is then read once for several bands, as long as four
  // blocks per SM remain
  int groups = (f.nbc + 3) / 4;
  while (groups < f.nbc && (int64_t)blocks * f.nk * groups < 4 * 148) ++groups;
  const int bpb = (f.nbc + groups - 1) / groups;
  dim3 g(blocks, (f.nbc + bpb - 1) / bpb, f.nk);
  constexpr size_t smem = C::R2 == 1 ? 0 : C::smem_strided + (size_t)C::R1 * C::NT * sizeof(cplx<T>);
  if (smem > 48 * 1024) {
    const cudaError_t e = allow_smem(k_pencil_vloc<T, N>);
    if (e != cudaSuccess) return e;
  }
  return launch_chained(k_pencil_vloc<T, N>, g, C::NT, smem, st, f, bpb);
}

template <typename T, int N> cudaError_t launch_density(const FftRun<T>& f, cudaStream_t st) {
  using C = AxisCfg<T, N>;
  dim3 g((f.n1 * f.n2 + C::PB - 1) / C::PB, f.ngrp, f.nk);
  if (2 * C::smem_strided > 48 * 1024) {
    const cudaError_t e = allow_smem(k_pencil_density<T, N>);
    if (e != cudaSuccess) return e;
  }
  return launch_chained(k_pencil_density<T, N>, g, C::NT, 2 * C::smem_strided, st, f);
}

}  // namespace fft_detail

}  // namespace gwb
