// Complex float64 products on the double-precision tensor instruction
// (mma.sync.m8n8k4.f64; tcgen05 has no float64 kind).
//
//   k_zmma_nh  part[s][b][i][j] = sum_{g in slice s} A[b][i][g] conj(B[b][j][g])
//              (rows contiguous in g: projector contraction, subspace, Gram and
//              projection products of the solver)
//   k_zmma_nn  out[b][i][g] += sum_q A[b][i][q] B[b][q][g]
//              (nonlocal update; for the generalized apply also
//              s[b][i][g] = (c + sum_q A2[b][i][q] B[b][q][g]) on the sphere)
//
// A complex product is four real ones on fragments that one 16-byte
// shared-memory load brings as (re, im). One instruction does 256 FMAs from
// three operand loads of one double per lane: the same tile on the FMA pipe
// reads two operands from shared memory per 2 x 2 outputs and issues 8x the
// instructions, which held these products at 10-14 TFLOP/s of the 37 the chip
// has in float64. A warp owns one 8-column tile and all TM rows of the block,
// so each B fragment is loaded once and there are 2 TM / 8 independent
// accumulation chains. Operands arrive by cp.async in 8-wide K steps, three
// stages deep.
//
// The tensor instruction rounds after every FMA, twice per complex term where a
// product rounded first costs one addition, so a chain of K terms from zero errs
// by sqrt(K) roundings of its sum. Chains are cut (and the sum taken over them)
// so that no product is further from exact than on the FMA pipe or in cuBLAS:
// after one K step in k_zmma_ab (24 x 256 x 96: 4.7e-16 uncut, 1.8e-16, cuBLAS
// 1.9e-16; 64 x 512 x 640: 12, 3.3, 6.0), after ZM_CHAIN in k_zmma_nh (24 x 24 x
// 100: 4.8e-16 with chains of 128 terms, 2.8e-16, FMA pipe 3.5e-16). The update is
// summed apart from the row it is added to, uncut up to ZM_UNCUT projectors (256:
// 8.3e-16, FMA pipe 9.2e-16; 512: 11 uncut, 3.7, 10; 864: 14, 4.3, 12); beyond, a
// cut per K step costs 5 % of an apply (400 projectors, 98 bands: 1051 -> 1112 us;
// per two steps 1137, whose live chains take a block per SM).
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"

namespace gwb {

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc, bool valid) {
  const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
  const int n = valid ? 16 : 0;  // 0: zero-fill, nothing read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(gsrc), "r"(n) : "memory");
}
// d += a b for one 8x8x4 tile: lane l holds a[l / 4][l % 4], b[l % 4][l / 4] and
// d[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

constexpr int ZM_K = 8;       // K step
constexpr int ZM_STAGES = 3;  // steps in flight
constexpr int ZM_CHAIN = 4;   // steps in one chain of k_zmma_nh
constexpr int ZM_UNCUT = 320;  // longest update summed in one chain

// Sums of a warp's 8 MT x 8 tile in chains of CHAIN steps (0: one chain): lane l
// holds rows 8 t + l / 4, columns 2 (l % 4) + {0, 1}.
template <int MT, int CHAIN> struct ZmmaSums {
  static constexpr int MS = CHAIN ? MT : 1;
  double re[MT][2] = {}, im[MT][2] = {}, sr[MS][2] = {}, si[MS][2] = {};
  // K step `step` of nsteps; a(t, kk), b(kk): this lane's elements of fragment kk (CONJ: product with conj(b)).
  template <bool CONJ, class FA, class FB>
  __device__ __forceinline__ void add(int step, int nsteps, FA&& a, FB&& b) {
#pragma unroll
    for (int kk = 0; kk < ZM_K; kk += 4) {
      const cplx<double> bv = b(kk);
#pragma unroll
      for (int t = 0; t < MT; ++t) {
        const cplx<double> av = a(t, kk);
        dmma(re[t], av.x, bv.x);
        dmma(im[t], av.y, bv.x);
        dmma(re[t], CONJ ? av.y : -av.y, bv.y);
        dmma(im[t], CONJ ? -av.x : av.x, bv.y);
      }
    }
    if constexpr (CHAIN > 0) {
      if (step % CHAIN == CHAIN - 1 || step == nsteps - 1) {
#pragma unroll
        for (int t = 0; t < MT; ++t)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            sr[t][e] += re[t][e];
            si[t][e] += im[t][e];
            re[t][e] = im[t][e] = 0.0;
          }
      }
    }
  }
  __device__ __forceinline__ cplx<double> at(int t, int e) const {
    return CHAIN ? mk<double>(sr[t % MS][e], si[t % MS][e]) : mk<double>(re[t][e], im[t][e]);
  }
};

// Row pitch of a K-contiguous tile: 12 elements of 16 bytes put the two rows of
// a quarter-warp (8 lanes: 2 rows x 4 k) 64 bytes apart modulo 128.
constexpr int ZM_PK = ZM_K + 4;

template <int TM, int TN> constexpr size_t zmma_nh_smem() {
  return (size_t)ZM_STAGES * (TM + TN) * ZM_PK * 16;
}

template <int TM, int TN>
__global__ void __launch_bounds__(TN * 4) k_zmma_nh(int M, int N, int K, int kslice,
                                                    const cplx<double>* __restrict__ A, int64_t lda, int64_t sA,
                                                    const cplx<double>* __restrict__ B, int64_t ldb, int64_t sB,
                                                    cplx<double>* __restrict__ part, int batch) {
  constexpr int NT = TN * 4, MT = TM / 8;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<double>* sm = reinterpret_cast<cplx<double>*>(smem_raw);  // [stage][TM + TN rows][ZM_PK]
  const int tilesN = (N + TN - 1) / TN;
  const int i0 = (blockIdx.x / tilesN) * TM, j0 = (blockIdx.x % tilesN) * TN;
  const int s = blockIdx.y, b = blockIdx.z;
  const cplx<double>* Ab = A + b * sA;
  const cplx<double>* Bb = B + b * sB;
  const int g0 = s * kslice, g1 = min(K, g0 + kslice);
  const int nsteps = (g1 - g0 + ZM_K - 1) / ZM_K;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;

  auto load = [&](int step) {
    if (step < nsteps) {
      const int gb = g0 + step * ZM_K;
      cplx<double>* st = sm + (size_t)(step % ZM_STAGES) * (TM + TN) * ZM_PK;
#pragma unroll
      for (int idx = tid; idx < (TM + TN) * ZM_K; idx += NT) {
        const int r = idx / ZM_K, kk = idx % ZM_K, g = gb + kk;
        const bool isA = r < TM;
        const int row = isA ? i0 + r : j0 + r - TM;
        const bool ok = row < (isA ? M : N) && g < g1;
        const cplx<double>* src = isA ? Ab + (int64_t)row * lda + g : Bb + (int64_t)row * ldb + g;
        cp_async16(st + r * ZM_PK + kk, ok ? src : Ab, ok);
      }
    }
    cp_async_commit();  // one group per step, empty past the end
  };

  ZmmaSums<MT, ZM_CHAIN> sum;
  chain_wait();
#pragma unroll
  for (int p = 0; p < ZM_STAGES - 1; ++p) load(p);
  for (int step = 0; step < nsteps; ++step) {
    cp_async_wait<ZM_STAGES - 2>();
    __syncthreads();  // this step has landed for all; the stage refilled next is read by none
    load(step + ZM_STAGES - 1);
    const cplx<double>* st = sm + (size_t)(step % ZM_STAGES) * (TM + TN) * ZM_PK;
    const cplx<double>* sa = st + (lane >> 2) * ZM_PK + (lane & 3);
    const cplx<double>* sb = st + (TM + w * 8 + (lane >> 2)) * ZM_PK + (lane & 3);
    sum.template add<true>(step, nsteps, [&](int t, int kk) { return sa[t * 8 * ZM_PK + kk]; },
                           [&](int kk) { return sb[kk]; });
  }
  cp_async_wait<0>();
  cplx<double>* P = part + ((int64_t)s * batch + b) * M * N;
  const int j = j0 + w * 8 + 2 * (lane & 3);
#pragma unroll
  for (int t = 0; t < MT; ++t) {
    const int i = i0 + t * 8 + (lane >> 2);
    if (i < M) {
      if (j < N) P[(int64_t)i * N + j] = sum.at(t, 0);
      if (j + 1 < N) P[(int64_t)i * N + j + 1] = sum.at(t, 1);
    }
  }
}

// Tile edge of M or N that costs least: padded extent plus 8 per tile for what
// a tile reloads of the other operand.
constexpr int zmma_edge(int64_t n, int most) {
  int best = 8;
  int64_t cost = -1;
  for (int t : {8, 16, 24, 32, 64}) {
    if (t > most) break;
    const int64_t c = (n + t - 1) / t * (t + 8);
    if (cost < 0 || c <= cost) cost = c, best = t;
  }
  return best;
}

// Launch of k_zmma_nh over ns slices of kslice (a multiple of ZM_K).
cudaError_t zmma_nh(int M, int N, int K, int kslice, int ns, const cplx<double>* A, int64_t lda, int64_t sA,
                    const cplx<double>* B, int64_t ldb, int64_t sB, cplx<double>* part, int batch, cudaStream_t st);
// Slices of K that give about target_blocks blocks of four warps, at most cap;
// *kslice is the slice length.
int zmma_nh_slices(int M, int N, int K, int batch, int64_t cap, int target_blocks, int* kslice);

// out_h += A P (and, with A2, out_s = (c + A2 P) on the sphere, 0 in the padding);
// A, A2: (batch, nb, K), P: (batch, K, N), rows of c / out_h / out_s N long.
cudaError_t zmma_nn(int nb, int N, int K, const cplx<double>* A, const cplx<double>* A2, const cplx<double>* P,
                    const cplx<double>* c, int64_t ck, cplx<double>* out_h, int64_t hk, cplx<double>* out_s, int64_t sk,
                    const int* npw_k, int batch, cudaStream_t st);

// C = alpha op(A) B + beta C with few rows: op(A) (M x K; TA: A is K x M), B (K x N),
// C (M x N), row-major, batched by strides. C is not read where beta = 0.
cudaError_t zmma_ab(bool TA, int M, int N, int K, cplx<double> alpha, const cplx<double>* A, int64_t lda, int64_t sA,
                    const cplx<double>* B, int64_t ldb, int64_t sB, cplx<double> beta, cplx<double>* C, int64_t ldc,
                    int64_t sC, int batch, cudaStream_t st);

}  // namespace gwb
