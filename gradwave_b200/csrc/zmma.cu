// Launch rules of the float64 tensor-instruction products (zmma.cuh) and the
// nonlocal update kernel.
#include <algorithm>

#include "zmma.cuh"

namespace gwb {

namespace {

// out tile: TM rows x 64 columns, one 8-column tile per warp. The rows are the
// nb rows of out_h, followed by the nb rows of out_s in the generalized apply.
constexpr int ZN_TN = 64;
// Row pitch of the P tile: 66 elements put the 4 k x 2 columns of a quarter-warp
// on distinct banks.
constexpr int ZN_PN = ZN_TN + 2;

template <int TM> constexpr size_t zmma_nn_smem() {
  return (size_t)ZM_STAGES * (TM * ZM_PK + ZM_K * ZN_PN) * 16;
}

template <int TM, bool HS, int CHAIN>
__global__ void __launch_bounds__(ZN_TN * 4) k_zmma_nn(int nb, int N, int K, const cplx<double>* __restrict__ A,
                                                       const cplx<double>* __restrict__ A2,
                                                       const cplx<double>* __restrict__ P,
                                                       const cplx<double>* __restrict__ c, int64_t ck,
                                                       cplx<double>* __restrict__ out_h, int64_t hk,
                                                       cplx<double>* __restrict__ out_s, int64_t sk,
                                                       const int* __restrict__ npw_k) {
  constexpr int NT = ZN_TN * 4, MT = TM / 8, STAGE = TM * ZM_PK + ZM_K * ZN_PN;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<double>* sm = reinterpret_cast<cplx<double>*>(smem_raw);
  const int rows = HS ? 2 * nb : nb;
  const int n0 = blockIdx.x * ZN_TN, i0 = blockIdx.y * TM, k = blockIdx.z;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int npw = HS ? npw_k[k] : N;
  const cplx<double>* Pk = P + (int64_t)k * K * N;
  const int nsteps = (K + ZM_K - 1) / ZM_K;

  auto load = [&](int step) {
    if (step < nsteps) {
      const int q0 = step * ZM_K;
      cplx<double>* st = sm + (size_t)(step % ZM_STAGES) * STAGE;
#pragma unroll
      for (int idx = tid; idx < TM * ZM_K; idx += NT) {
        const int r = idx / ZM_K, qq = idx % ZM_K, i = i0 + r, q = q0 + qq;
        const bool ok = i < rows && q < K;
        const cplx<double>* src = HS && i >= nb ? A2 + ((int64_t)k * nb + i - nb) * K + q
                                                : A + ((int64_t)k * nb + i) * K + q;
        cp_async16(st + r * ZM_PK + qq, ok ? src : A, ok);
      }
#pragma unroll
      for (int idx = tid; idx < ZM_K * ZN_TN; idx += NT) {
        const int qq = idx / ZN_TN, nn = idx % ZN_TN, q = q0 + qq, n = n0 + nn;
        const bool ok = q < K && n < N;
        cp_async16(st + TM * ZM_PK + qq * ZN_PN + nn, ok ? Pk + (int64_t)q * N + n : Pk, ok);
      }
    }
    cp_async_commit();
  };
  chain_wait();
  c = after_wait(c);
  out_h = after_wait(out_h);  // without projectors the kernel just before this one wrote it
#pragma unroll
  for (int p = 0; p < ZM_STAGES - 1; ++p) load(p);

  const int n = n0 + w * 8 + 2 * (lane & 3);
  ZmmaSums<MT, CHAIN> sum;
  for (int step = 0; step < nsteps; ++step) {
    cp_async_wait<ZM_STAGES - 2>();
    __syncthreads();
    load(step + ZM_STAGES - 1);
    const cplx<double>* st = sm + (size_t)(step % ZM_STAGES) * STAGE;
    const cplx<double>* sa = st + (lane >> 2) * ZM_PK + (lane & 3);
    const cplx<double>* sp = st + TM * ZM_PK + (lane & 3) * ZN_PN + w * 8 + (lane >> 2);
    sum.template add<false>(step, nsteps, [&](int t, int kk) { return sa[t * 8 * ZM_PK + kk]; },
                            [&](int kk) { return sp[kk * ZN_PN]; });
  }
  cp_async_wait<0>();
#pragma unroll
  for (int t = 0; t < MT; ++t) {
    const int i = i0 + t * 8 + (lane >> 2);
    if (i >= rows) continue;
    const bool sr = HS && i >= nb;
    cplx<double>* dst = sr ? out_s + (int64_t)k * sk + (int64_t)(i - nb) * N : out_h + (int64_t)k * hk + (int64_t)i * N;
    const cplx<double>* src = sr ? c + (int64_t)k * ck + (int64_t)(i - nb) * N : dst;
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (n + e < N)
        dst[n + e] = sr && n + e >= npw ? mk<double>(0.0, 0.0) : src[n + e] + sum.at(t, e);
  }
}

// The same tiles for the solver's short products (triangular transforms,
// projections, Ritz vectors: few rows, long rows of B).
template <int TM, bool TA>
__global__ void __launch_bounds__(ZN_TN * 4) k_zmma_ab(int M, int N, int K, cplx<double> alpha,
                                                       const cplx<double>* __restrict__ A, int64_t lda, int64_t sA,
                                                       const cplx<double>* __restrict__ B, int64_t ldb, int64_t sB,
                                                       cplx<double> beta, cplx<double>* C, int64_t ldc, int64_t sC) {
  constexpr int NT = ZN_TN * 4, MT = TM / 8, STAGE = TM * ZM_PK + ZM_K * ZN_PN;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<double>* sm = reinterpret_cast<cplx<double>*>(smem_raw);
  const int n0 = blockIdx.x * ZN_TN, i0 = blockIdx.y * TM;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const cplx<double>* Ab = A + blockIdx.z * sA;
  const cplx<double>* Bb = B + blockIdx.z * sB;
  cplx<double>* Cb = C + blockIdx.z * sC;
  const int nsteps = (K + ZM_K - 1) / ZM_K;

  auto load = [&](int step) {
    if (step < nsteps) {
      const int q0 = step * ZM_K;
      cplx<double>* st = sm + (size_t)(step % ZM_STAGES) * STAGE;
#pragma unroll
      for (int idx = tid; idx < TM * ZM_K; idx += NT) {
        const int r = TA ? idx % TM : idx / ZM_K, qq = TA ? idx / TM : idx % ZM_K, i = i0 + r, q = q0 + qq;
        const bool ok = i < M && q < K;
        const cplx<double>* src = TA ? Ab + (int64_t)q * lda + i : Ab + (int64_t)i * lda + q;
        cp_async16(st + r * ZM_PK + qq, ok ? src : Ab, ok);
      }
#pragma unroll
      for (int idx = tid; idx < ZM_K * ZN_TN; idx += NT) {
        const int qq = idx / ZN_TN, nn = idx % ZN_TN, q = q0 + qq, n = n0 + nn;
        const bool ok = q < K && n < N;
        cp_async16(st + TM * ZM_PK + qq * ZN_PN + nn, ok ? Bb + (int64_t)q * ldb + n : Bb, ok);
      }
    }
    cp_async_commit();
  };
  chain_wait();
#pragma unroll
  for (int p = 0; p < ZM_STAGES - 1; ++p) load(p);
  ZmmaSums<MT, 1> sum;
  for (int step = 0; step < nsteps; ++step) {
    cp_async_wait<ZM_STAGES - 2>();
    __syncthreads();
    load(step + ZM_STAGES - 1);
    const cplx<double>* st = sm + (size_t)(step % ZM_STAGES) * STAGE;
    const cplx<double>* sa = st + (lane >> 2) * ZM_PK + (lane & 3);
    const cplx<double>* sb = st + TM * ZM_PK + (lane & 3) * ZN_PN + w * 8 + (lane >> 2);
    sum.template add<false>(step, nsteps, [&](int t, int kk) { return sa[t * 8 * ZM_PK + kk]; },
                            [&](int kk) { return sb[kk * ZN_PN]; });
  }
  cp_async_wait<0>();
  const int n = n0 + w * 8 + 2 * (lane & 3);
  const bool add = beta.x != 0.0 || beta.y != 0.0;
#pragma unroll
  for (int t = 0; t < MT; ++t) {
    const int i = i0 + t * 8 + (lane >> 2);
    if (i >= M) continue;
    cplx<double>* dst = Cb + (int64_t)i * ldc;
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (n + e < N) {
        const cplx<double> v = alpha * sum.at(t, e);
        dst[n + e] = add ? v + beta * dst[n + e] : v;
      }
  }
}

}  // namespace

cudaError_t zmma_ab(bool TA, int M, int N, int K, cplx<double> alpha, const cplx<double>* A, int64_t lda, int64_t sA,
                    const cplx<double>* B, int64_t ldb, int64_t sB, cplx<double> beta, cplx<double>* C, int64_t ldc,
                    int64_t sC, int batch, cudaStream_t st) {
  const int TM = zmma_edge(M, 32);
  const dim3 grid((unsigned)((N + ZN_TN - 1) / ZN_TN), (unsigned)((M + TM - 1) / TM), batch);
#define GWB_ZA_CASE(tm)                                                                                          \
  if (TM == tm)                                                                                                  \
    return launch_chained(TA ? k_zmma_ab<tm, true> : k_zmma_ab<tm, false>, grid, ZN_TN * 4, zmma_nn_smem<tm>(), st, M, \
                          N, K, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC);
  GWB_ZA_CASE(8) GWB_ZA_CASE(16) GWB_ZA_CASE(24) GWB_ZA_CASE(32)
#undef GWB_ZA_CASE
  return cudaErrorInvalidValue;
}

int zmma_nh_slices(int M, int N, int K, int batch, int64_t cap, int target_blocks, int* kslice) {
  const int TM = zmma_edge(M, 32), TN = zmma_edge(N, 64);
  const int64_t tiles = (int64_t)((M + TM - 1) / TM) * ((N + TN - 1) / TN) * batch;
  int64_t want = ((int64_t)target_blocks * std::max(1, 32 / TN) + tiles - 1) / tiles;
  // slices at least 128 long (their sum is read back), 64 while there is less than a block per SM
  const int64_t most = std::max<int64_t>(K / 128, std::min<int64_t>(K / 64, 148 / tiles));
  want = std::max<int64_t>(1, std::min<int64_t>({want, cap, most}));
  *kslice = (int)std::max<int64_t>(ZM_K, ((K + want - 1) / want + ZM_K - 1) / ZM_K * ZM_K);
  return std::max(1, (K + *kslice - 1) / *kslice);
}

cudaError_t zmma_nh(int M, int N, int K, int kslice, int ns, const cplx<double>* A, int64_t lda, int64_t sA,
                    const cplx<double>* B, int64_t ldb, int64_t sB, cplx<double>* part, int batch, cudaStream_t st) {
  const int TM = zmma_edge(M, 32), TN = zmma_edge(N, 64);
  const dim3 grid((unsigned)(((M + TM - 1) / TM) * ((N + TN - 1) / TN)), ns, batch);
#define GWB_ZM_CASE(tm, tn)                                                                               \
  if (TM == tm && TN == tn) {                                                                             \
    constexpr size_t smem = zmma_nh_smem<tm, tn>();                                                       \
    if (smem > 48 * 1024) {                                                                               \
      const cudaError_t e = allow_smem(k_zmma_nh<tm, tn>);                                                \
      if (e != cudaSuccess) return e;                                                                     \
    }                                                                                                     \
    return launch_chained(k_zmma_nh<tm, tn>, grid, tn * 4, smem, st, M, N, K, kslice, A, lda, sA, B, ldb, sB, \
                          part, batch);                                                                   \
  }
#define GWB_ZM_ROW(tm) GWB_ZM_CASE(tm, 8) GWB_ZM_CASE(tm, 16) GWB_ZM_CASE(tm, 24) GWB_ZM_CASE(tm, 32) GWB_ZM_CASE(tm, 64)
  GWB_ZM_ROW(8) GWB_ZM_ROW(16) GWB_ZM_ROW(24) GWB_ZM_ROW(32)
#undef GWB_ZM_ROW
#undef GWB_ZM_CASE
  return cudaErrorInvalidValue;
}

cudaError_t zmma_nn(int nb, int N, int K, const cplx<double>* A, const cplx<double>* A2, const cplx<double>* P,
                    const cplx<double>* c, int64_t ck, cplx<double>* out_h, int64_t hk, cplx<double>* out_s, int64_t sk,
                    const int* npw_k, int batch, cudaStream_t st) {
  const int rows = A2 ? 2 * nb : nb;
  const int TM = zmma_edge(rows, 32);
  const bool uncut = K <= ZM_UNCUT;
  const dim3 grid((unsigned)((N + ZN_TN - 1) / ZN_TN), (unsigned)((rows + TM - 1) / TM), batch);
#define GWB_ZN_CASE(tm)                                                                                            \
  if (TM == tm) {                                                                                                  \
    auto* kern = A2 ? (uncut ? k_zmma_nn<tm, true, 0> : k_zmma_nn<tm, true, 1>)                             \
                    : (uncut ? k_zmma_nn<tm, false, 0> : k_zmma_nn<tm, false, 1>);                          \
    return launch_chained(kern, grid, ZN_TN * 4, zmma_nn_smem<tm>(), st, nb, N, K, A, A2, P, c, ck, out_h, hk,     \
                          out_s, sk, npw_k);                                                                       \
  }
  GWB_ZN_CASE(8) GWB_ZN_CASE(16) GWB_ZN_CASE(24) GWB_ZN_CASE(32)
#undef GWB_ZN_CASE
  return cudaErrorInvalidValue;
}

}  // namespace gwb
