// Batched plane-wave Hamiltonian apply H c = T c + V_loc c + sum p D <p|c>
// for all k-points and bands in a few launches (sm_100a).
//
// Local term (replaces gradwave core/batch.py:405-428). The sphere of each k
// occupies Miller indices |m_a| <= M_a of a box n0 x n1 x n2, so only
// L_a = 2 M_a + 1 planes/rows/columns per axis ever hold data, and of the rows
// (j0, i1) only those of a disc. Five launches per chunk of bands
// (fft_axis.cuh): axis 2 of the disc's rows, axis 1 of the occupied planes,
// axis 0 with the product with v(r)/N and back, axis 1, axis 2 with the
// kinetic term. The bands are processed in chunks that bound the scratch (W and
// W2).
//
// Nonlocal term (replaces gradwave core/batch.py:499-500 and becp_b :590-595):
//   K4 becp_partial   becp partial sums conj(p) . c over a slice of G
//   K5 becp_reduce_d  sum of slices, times D  -> bd (nk, nb, nproj)
//   K6 nl_add         out += bd . p
// (float64 arithmetic on complex128 rows: K4 and K6 on the float64 tensor
// instruction, zmma.cuh)
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <atomic>
#include <memory>
#include <new>
#include <string>
#include <vector>

#include "common.cuh"
#include "device_pool.cuh"
#include "fft_axis.cuh"
#include "zmma.cuh"

namespace gwb {

static thread_local std::string g_last_error;
void set_error(const std::string& msg) { g_last_error = msg; }
static std::atomic<unsigned long long> g_launches{0};
void count_launches(int n) { g_launches.fetch_add((unsigned long long)n, std::memory_order_relaxed); }

struct FftGeom {
  int n[3];
  int M[3];  // max |Miller index| per axis over all k (compact row map)
  int L[3];  // occupied extent per axis (2M+1, capped at n)
  int nrow;  // row slots (j0, i1) per k, the most of any k
};

}  // namespace gwb

struct gwb_ham {
  int device = 0;
  int nk = 0, npw_max = 0, nproj = 0;
  gwb::FftGeom g{};
  std::vector<int64_t> npw_host;
  // device tables
  int* d_npw = nullptr;
  int* d_map = nullptr;    // (nk, nrow, n2) sphere index of each row point, -1: none
  int* d_rowof = nullptr;  // (nk, L0, n1) row slot of (j0, i1), -1: none
  int* d_dup = nullptr;    // (ndup, 3) k, slot, other slot of the same box cell
  int ndup = 0;
  double* d_t64 = nullptr;
  float* d_t32 = nullptr;
  double* d_v64 = nullptr;  // v(r)/N
  float* d_v32 = nullptr;
  gwb::cplx<double>* d_p64 = nullptr;
  gwb::cplx<float>* d_p32 = nullptr;
  double* d_d64 = nullptr;
  float* d_d32 = nullptr;
  gwb::ColumnLists d_cols, q_cols;  // nonzeros of D and q per column
  double* d_q64 = nullptr;  // augmentation q_pq of the overlap S (USPP/PAW), when set
  float* d_q32 = nullptr;
  gwb::cplx<double>* d_tw64[3] = {nullptr, nullptr, nullptr};
  gwb::cplx<float>* d_tw32[3] = {nullptr, nullptr, nullptr};
  // scratch
  gwb::ChunkScratch W;   // planes of a band chunk, then its rows
  bool counted = false;  // among its device's live handles (gwb_ham_create completed)
  void* d_part = nullptr;  // becp partials
  size_t part_bytes = 0;
  void* d_bd = nullptr;  // becp * D
  size_t bd_bytes = 0;
  void* d_bq = nullptr;  // becp * q (overlap apply)
  size_t bq_bytes = 0;
  // tensor-core nonlocal term (float32 applies of complex128 blocks)
  void* d_pplanes = nullptr;  // BF16 planes of P: (nk, 4, nproj, ldp)
  size_t pplanes_bytes = 0;
  bool pplanes_ok = false;
  void* d_cplanes = nullptr;  // BF16 planes of the input rows: (nk, 4, nb, ldp)
  size_t cplanes_bytes = 0;
  void* d_becp = nullptr;  // becp (nk, nb, nproj) complex128
  size_t becp_bytes = 0;
  void* d_bdplanes = nullptr;  // BF16 planes of becp D: (nk, 4, nb, ldq)
  size_t bdplanes_bytes = 0;
  void* d_tcwork = nullptr;  // split-K partial sums
  size_t tcwork_bytes = 0;
  int* d_tcstatus = nullptr;  // pipeline-wait timeouts of the tensor-core products
  double* d_rhok = nullptr;  // density accumulators, one box per k
  size_t rhok_bytes = 0;
  bool have_t = false, have_v = false, have_p = false, have_q = false;
  // tuning (gwb_ham_set_tuning; 0 = the built-in rule)
  size_t w_budget = 0;   // bytes of FFT scratch W per band chunk
  int nl_target = 0;     // CTAs the G-sliced becp contraction aims for
};

namespace gwb {

static bool axis_ok(int n) {
  if (n < 2 || n > 128) return false;
  for (int p : {2, 3, 5, 7})
    while (n % p == 0) n /= p;
  return n == 1;
}

// exp(2 pi i m / n), the angle reduced to an eighth of a turn exactly and taken in
// extended precision: cos and sin of a rounded 2 pi m / n are off by up to 8e-16.
static cplx<double> unit_root(int m, int n) {
  const int q = (8 * m + n) / (2 * n);  // nearest quarter turn
  const long double x = 3.14159265358979323846264338327950288L * (4 * m - q * n) / (2 * n);
  const double c = (double)std::cos(x), s = (double)std::sin(x);
  const cplx<double> r[4] = {mk<double>(c, s), mk<double>(-s, c), mk<double>(-c, -s), mk<double>(s, -c)};
  return r[q % 4];
}

// Scratch of one band chunk. A float64 96^3 Gamma apply of 240 rows takes 8.2 ms
// at 48 MB (L2 sized), 8.0 at 96 to 192, 7.7 at 512, 7.5 at 1024: launch ramps and
// last waves weigh more than L2 misses, and past 512 MB little is left.
constexpr long kWBudgetMB = 512, kWBudgetLowMB = 48;

static size_t w_budget_bytes() {
  const char* s = std::getenv("GWB_W_BUDGET_MB");
  long mb = s ? std::atol(s) : kWBudgetMB;
  if (mb < 1) mb = 1;
  return (size_t)mb << 20;
}

// rho[r] = scale sum_s rho_s[s][r] over the nsum accumulators (k, band group), in order.
__global__ void k_density_sum(int nsum, int64_t N, const double* __restrict__ rho_s, double scale,
                              double* __restrict__ rho) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x) {
    double a = 0.0;
    for (int k = 0; k < nsum; ++k) a += rho_s[(int64_t)k * N + i];
    rho[i] = scale * a;
  }
}

// Sphere slots that name the box cell of another slot of the same k (not met
// in a sphere of distinct G): the transforms read and write the last such slot,
// the others get its local term with their own kinetic term here.
template <typename T, typename SIO>
__global__ void k_duplicate_slots(const int* __restrict__ dup, int ndup, const SIO* __restrict__ c, int64_t ck,
                                  SIO* __restrict__ out, int64_t ok, const T* __restrict__ t, int nb, int npw_max) {
  const int total = ndup * nb;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int* d = dup + 3 * (i / nb);
    const int b = i % nb, k = d[0], g = d[1], h = d[2];
    const size_t ci = (size_t)k * ck + (size_t)b * npw_max, oi = (size_t)k * ok + (size_t)b * npw_max;
    const T* tk = t + (size_t)k * npw_max;
    const cplx<T> local = ld<T>(out, oi + h) - scale(ld<T>(c, ci + h), tk[h]);
    st(out, oi + g, local + scale(ld<T>(c, ci + g), tk[g]));
  }
}

// ---------------------------------------------------------------------------
// Nonlocal term. Tiles: TB bands x TP projectors, G slices of TG.
constexpr int NL_TB = 16, NL_TP = 32, NL_TG = 32;

// K4: part[s][k][b][p] = sum_{g in slice s} conj(P[k][p][g]) c[k][b][g].
// The next step's tiles are loaded into registers while this step multiplies
// out of shared memory (one barrier pair per step).
template <typename T, typename SIO>
__global__ void __launch_bounds__(256) k_becp_partial(const SIO* __restrict__ c,
                                                      const cplx<T>* __restrict__ P,
                                                      cplx<T>* __restrict__ part, int nk, int nb,
                                                      int nproj, int npw_max, int gslice, int64_t ck) {
  constexpr int LC = NL_TB * NL_TG / 256, LP = NL_TP * NL_TG / 256;  // elements per thread per step
  __shared__ cplx<T> sc[NL_TB][NL_TG + 1];
  __shared__ cplx<T> sp[NL_TP][NL_TG + 1];
  const int pt = blockIdx.x, bt = blockIdx.y;
  const int k = blockIdx.z % nk, s = blockIdx.z / nk;
  const int tid = threadIdx.x;
  const int lb = tid / 16, lp = tid % 16;  // each thread: band lb, projectors lp and lp+16
  cplx<T> acc0 = mk<T>(0, 0), acc1 = mk<T>(0, 0);
  const int g_begin = s * gslice, g_end = min(npw_max, g_begin + gslice);
  cplx<T> rc[LC], rp[LP];
  auto fetch = [&](int gb) {
#pragma unroll
    for (int q = 0; q < LC; ++q) {
      const int i = tid + 256 * q, bb = i / NL_TG, gg = i % NL_TG;
      const int b = bt * NL_TB + bb, gi = gb + gg;
      rc[q] = (b < nb && gi < g_end) ? ld<T>(c, (size_t)k * ck + (size_t)b * npw_max + gi) : mk<T>(0, 0);
    }
#pragma unroll
    for (int q = 0; q < LP; ++q) {
      const int i = tid + 256 * q, pp = i / NL_TG, gg = i % NL_TG;
      const int p = pt * NL_TP + pp, gi = gb + gg;
      rp[q] = (p < nproj && gi < g_end) ? P[((size_t)k * nproj + p) * npw_max + gi] : mk<T>(0, 0);
    }
  };
  chain_wait();
  c = after_wait(c);
  if (g_begin < g_end) fetch(g_begin);
  for (int gb = g_begin; gb < g_end; gb += NL_TG) {
#pragma unroll
    for (int q = 0; q < LC; ++q) {
      const int i = tid + 256 * q;
      sc[i / NL_TG][i % NL_TG] = rc[q];
    }
#pragma unroll
    for (int q = 0; q < LP; ++q) {
      const int i = tid + 256 * q;
      sp[i / NL_TG][i % NL_TG] = rp[q];
    }
    __syncthreads();
    if (gb + NL_TG < g_end) fetch(gb + NL_TG);
#pragma unroll 8
    for (int gg = 0; gg < NL_TG; ++gg) {
      const cplx<T> cv = sc[lb][gg];
      acc0 = acc0 + conj_mul(sp[lp][gg], cv);
      acc1 = acc1 + conj_mul(sp[lp + 16][gg], cv);
    }
    __syncthreads();
  }
  const int b = bt * NL_TB + lb;
  if (b < nb) {
    const size_t row = (((size_t)s * nk + k) * nb + b) * nproj;
    const int p0 = pt * NL_TP + lp, p1 = p0 + 16;
    if (p0 < nproj) part[row + p0] = acc0;
    if (p1 < nproj) part[row + p1] = acc1;
  }
}

// Sum of the slice partials of one (k, band) into becp (shared memory): the
// slices are split over the threads (projector p, slice group) and combined in
// a fixed order (deterministic).
template <typename T>
__device__ __forceinline__ void sum_slices(const cplx<T>* part, cplx<T>* becp, cplx<T>* grp, size_t stride,
                                           size_t row, int nproj, int nslice) {
  const int ngrp = max(1, (int)blockDim.x / nproj);
  chain_wait();
  part = after_wait(part);
  for (int idx = threadIdx.x; idx < nproj * ngrp; idx += blockDim.x) {
    const int p = idx % nproj, gq = idx / nproj;
    cplx<T> a = mk<T>(0, 0);
    for (int s = gq; s < nslice; s += ngrp) a = a + part[s * stride + row + p];
    grp[gq * nproj + p] = a;
  }
  __syncthreads();
  for (int p = threadIdx.x; p < nproj; p += blockDim.x) {
    cplx<T> a = mk<T>(0, 0);
    for (int gq = 0; gq < ngrp; ++gq) a = a + grp[gq * nproj + p];
    becp[p] = a;
  }
  __syncthreads();
}

// K5: bd[k][b][q] = sum_p (sum_s part[s][k][b][p]) D[p][q].
template <typename T>
__global__ void __launch_bounds__(128) k_becp_reduce_d(const cplx<T>* __restrict__ part, const T* __restrict__ D,
                                                       ColumnLists cols, cplx<T>* __restrict__ bd, int nk, int nb,
                                                       int nproj, int nslice) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* becp = reinterpret_cast<cplx<T>*>(smem_raw);  // nproj
  const size_t row = (size_t)blockIdx.x * nproj;         // blockIdx.x = k*nb + b
  sum_slices(part, becp, becp + nproj, (size_t)nk * nb * nproj, row, nproj, nslice);
  for (int q = threadIdx.x; q < nproj; q += blockDim.x) bd[row + q] = column_sum(cols, D, nproj, q, becp);
}

// K6: out[k][b][g] += sum_q bd[k][b][q] P[k][q][g]; tiles TB bands x 64 G.
template <typename T, typename SIO>
__global__ void __launch_bounds__(256) k_nl_add(const cplx<T>* __restrict__ bd,
                                                const cplx<T>* __restrict__ P,
                                                SIO* __restrict__ out, int nk, int nb, int nproj,
                                                int npw_max, int64_t ok) {
  constexpr int TGO = 64, TQ = 16;
  __shared__ cplx<T> sb[NL_TB][TQ];
  __shared__ cplx<T> sp[TQ][TGO];
  const int gt = blockIdx.x, bt = blockIdx.y, k = blockIdx.z;
  const int tid = threadIdx.x;
  const int lg = tid % TGO, lb0 = tid / TGO;  // 4 band groups x 64 g; each thread 4 bands
  cplx<T> acc[4];
  const int gi_o = gt * TGO + lg;
  chain_wait();
  bd = after_wait(bd);
  out = after_wait(out);
#pragma unroll
  for (int i = 0; i < 4; ++i) {  // the output rows first: their loads overlap the tile staging below
    const int b = bt * NL_TB + lb0 * 4 + i;
    acc[i] = (gi_o < npw_max && b < nb) ? ld<T>(out, (size_t)k * ok + (size_t)b * npw_max + gi_o) : mk<T>(0, 0);
  }
  for (int q0 = 0; q0 < nproj; q0 += TQ) {
    for (int i = tid; i < NL_TB * TQ; i += blockDim.x) {
      const int bb = i / TQ, qq = i % TQ;
      const int b = bt * NL_TB + bb, q = q0 + qq;
      sb[bb][qq] = (b < nb && q < nproj) ? bd[((size_t)k * nb + b) * nproj + q] : mk<T>(0, 0);
    }
    for (int i = tid; i < TQ * TGO; i += blockDim.x) {
      const int qq = i / TGO, gg = i % TGO;
      const int q = q0 + qq, gi = gt * TGO + gg;
      sp[qq][gg] = (q < nproj && gi < npw_max) ? P[((size_t)k * nproj + q) * npw_max + gi] : mk<T>(0, 0);
    }
    __syncthreads();
#pragma unroll
    for (int qq = 0; qq < TQ; ++qq) {
      const cplx<T> pv = sp[qq][lg];
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i] = acc[i] + sb[lb0 * 4 + i][qq] * pv;
    }
    __syncthreads();
  }
  if (gi_o < npw_max) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int b = bt * NL_TB + lb0 * 4 + i;
      if (b < nb) st(out, (size_t)k * ok + (size_t)b * npw_max + gi_o, acc[i]);
    }
  }
}

// K5 of the generalized apply: one pass over the slice partials gives both
// bd = becp D (H) and bq = becp q (S).
template <typename T>
__global__ void __launch_bounds__(128) k_becp_reduce_dq(const cplx<T>* __restrict__ part, const T* __restrict__ D,
                                                        ColumnLists dcols, const T* __restrict__ Q, ColumnLists qcols,
                                                        cplx<T>* __restrict__ bd, cplx<T>* __restrict__ bq, int nk,
                                                        int nb, int nproj, int nslice) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* becp = reinterpret_cast<cplx<T>*>(smem_raw);
  const size_t row = (size_t)blockIdx.x * nproj;
  sum_slices(part, becp, becp + nproj, (size_t)nk * nb * nproj, row, nproj, nslice);
  for (int q = threadIdx.x; q < nproj; q += blockDim.x) {
    bd[row + q] = column_sum(dcols, D, nproj, q, becp);
    bq[row + q] = column_sum(qcols, Q, nproj, q, becp);
  }
}

// K6 of the generalized apply: each projector tile is read once for both
// outputs, out_h += bd P and out_s = (c + bq P) on the sphere, 0 in the
// padding (the overlap's mask).
template <typename T, typename SIO>
__global__ void __launch_bounds__(256) k_nl_add_hs(const cplx<T>* __restrict__ bd, const cplx<T>* __restrict__ bq,
                                                   const cplx<T>* __restrict__ P, const SIO* __restrict__ c,
                                                   int64_t ck, SIO* __restrict__ out_h, int64_t ohk,
                                                   SIO* __restrict__ out_s, int64_t osk,
                                                   const int* __restrict__ npw_k, int nk, int nb, int nproj,
                                                   int npw_max) {
  constexpr int TGO = 64, TQ = 16;
  __shared__ cplx<T> sb[NL_TB][TQ];
  __shared__ cplx<T> sq[NL_TB][TQ];
  __shared__ cplx<T> sp[TQ][TGO];
  const int gt = blockIdx.x, bt = blockIdx.y, k = blockIdx.z;
  const int tid = threadIdx.x;
  const int lg = tid % TGO, lb0 = tid / TGO;
  const int gi_o = gt * TGO + lg;
  const bool on_sphere = gi_o < npw_k[k];
  cplx<T> ah[4], as[4];
  chain_wait();
  bd = after_wait(bd);
  bq = after_wait(bq);
  c = after_wait(c);
  out_h = after_wait(out_h);  // without projectors the kernel just before this one wrote it
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int b = bt * NL_TB + lb0 * 4 + i;
    const bool ok = gi_o < npw_max && b < nb;
    ah[i] = ok ? ld<T>(out_h, (size_t)k * ohk + (size_t)b * npw_max + gi_o) : mk<T>(0, 0);
    as[i] = (ok && on_sphere) ? ld<T>(c, (size_t)k * ck + (size_t)b * npw_max + gi_o) : mk<T>(0, 0);
  }
  for (int q0 = 0; q0 < nproj; q0 += TQ) {
    for (int i = tid; i < NL_TB * TQ; i += blockDim.x) {
      const int bb = i / TQ, qq = i % TQ;
      const int b = bt * NL_TB + bb, q = q0 + qq;
      const bool ok = b < nb && q < nproj;
      sb[bb][qq] = ok ? bd[((size_t)k * nb + b) * nproj + q] : mk<T>(0, 0);
      sq[bb][qq] = ok ? bq[((size_t)k * nb + b) * nproj + q] : mk<T>(0, 0);
    }
    for (int i = tid; i < TQ * TGO; i += blockDim.x) {
      const int qq = i / TGO, gg = i % TGO;
      const int q = q0 + qq, gi = gt * TGO + gg;
      sp[qq][gg] = (q < nproj && gi < npw_max) ? P[((size_t)k * nproj + q) * npw_max + gi] : mk<T>(0, 0);
    }
    __syncthreads();
#pragma unroll
    for (int qq = 0; qq < TQ; ++qq) {
      const cplx<T> pv = sp[qq][lg];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        ah[i] = ah[i] + sb[lb0 * 4 + i][qq] * pv;
        as[i] = as[i] + sq[lb0 * 4 + i][qq] * pv;
      }
    }
    __syncthreads();
  }
  if (gi_o < npw_max) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int b = bt * NL_TB + lb0 * 4 + i;
      if (b < nb) {
        st(out_h, (size_t)k * ohk + (size_t)b * npw_max + gi_o, ah[i]);
        st(out_s, (size_t)k * osk + (size_t)b * npw_max + gi_o, on_sphere ? as[i] : mk<T>(0, 0));
      }
    }
  }
}

template <typename T> __global__ void k_scale_copy(const double* src, T* dst, size_t n, double s) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < n) dst[i] = (T)(src[i] * s);
}
// Nonzeros of each column of the n x n matrix D, rows ascending.
__global__ void k_column_lists(const double* __restrict__ D, int n, int* __restrict__ cnt, int* __restrict__ idx) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  int c = 0;
#pragma unroll 8
  for (int p = 0; p < n; ++p)
    if (D[(size_t)p * n + q] != 0.0) idx[(size_t)c++ * n + q] = p;
  cnt[q] = c;
}

__global__ void k_c128_to_c64(const cplx<double>* src, cplx<float>* dst, size_t n) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < n) dst[i] = mk<float>((float)src[i].x, (float)src[i].y);
}

struct CudaMemory {
  static bool alloc(void** p, size_t bytes) {
    if (cudaMalloc(p, bytes) == cudaSuccess) return true;
    cudaGetLastError();
    return false;
  }
  static void free(void* p) { cudaFree(p); }
};
static DevicePool<CudaMemory> g_pool;

static int ensure_buf(const gwb_ham* h, void** p, size_t* have, size_t need) {
  if (g_pool.ensure(h->device, p, have, need)) return GWB_OK;
  set_error("device allocation of " + std::to_string(need) + " bytes failed");
  return GWB_ERR_ALLOC;
}

// G slices of the becp reduction: enough CTAs to fill the GPU (4 per SM)
// with every slice at least 256 plane waves long.
static int nl_slices(const gwb_ham* h, int nb) {
  const int tiles = ((h->nproj + NL_TP - 1) / NL_TP) * ((nb + NL_TB - 1) / NL_TB) * h->nk;
  const int target = h->nl_target > 0 ? h->nl_target : 4 * 148;
  const int want = (target + tiles - 1) / tiles;
  const int cap = std::max(1, h->npw_max / 256);
  return std::max(1, std::min(want, cap));
}

// Bands per chunk and the chunk's scratch (W: L0 planes, W2: the disc's rows).
static int chunk_scratch(gwb_ham* h, int nb, size_t es, int* nbc) {
  const FftGeom& g = h->g;
  const size_t per_band = (size_t)h->nk * ((size_t)g.L[0] * g.n[1] + g.nrow) * g.n[2] * es;
  *nbc = g_pool.chunk(h->device, h->W, nb, per_band, h->w_budget ? h->w_budget : w_budget_bytes(),
                      (size_t)kWBudgetLowMB << 20);
  if (*nbc) return GWB_OK;
  set_error("no device memory for the scratch of one band (" + std::to_string(per_band) + " bytes)");
  return GWB_ERR_ALLOC;
}

template <typename T> static FftRun<T> fft_run(const gwb_ham* h, int nbc) {
  const FftGeom& g = h->g;
  const bool dbl = sizeof(T) == 8;
  FftRun<T> f{};
  f.n0 = g.n[0], f.n1 = g.n[1], f.n2 = g.n[2];
  f.M0 = g.M[0], f.L0 = g.L[0], f.M2 = g.M[2];
  f.nk = h->nk, f.nrow = g.nrow, f.nbc = nbc, f.npw_max = h->npw_max;
  f.map = h->d_map, f.rowof = h->d_rowof, f.npw = h->d_npw;
  f.tw0 = dbl ? (const cplx<T>*)h->d_tw64[0] : (const cplx<T>*)h->d_tw32[0];
  f.tw1 = dbl ? (const cplx<T>*)h->d_tw64[1] : (const cplx<T>*)h->d_tw32[1];
  f.tw2 = dbl ? (const cplx<T>*)h->d_tw64[2] : (const cplx<T>*)h->d_tw32[2];
  f.v = dbl ? (const T*)h->d_v64 : (const T*)h->d_v32;
  f.t = dbl ? (const T*)h->d_t64 : (const T*)h->d_t32;
  f.W = (cplx<T>*)h->W.p;
  return f;
}

// rows' scratch of a chunk: behind its planes
template <typename T> static void place_rows(const gwb_ham* h, FftRun<T>* f) {
  f->W2 = f->W + (size_t)h->nk * f->nbc * f->L0 * f->n1 * f->n2;
}

int tc_becp_d_planes(int nk, int nb, int nproj, const cplx<double>* becp, const double* D, const ColumnLists& cols,
                     void* planes, int64_t ldq, cudaStream_t st);

// Projector counts from which the float32 apply of complex128 blocks runs its
// nonlocal term on the tensor cores (GWB_TC_NONLOCAL=0 keeps the CUDA-core
// kernels everywhere).
constexpr int TC_NONLOCAL_MIN_NPROJ = 128;

static bool tc_nonlocal_enabled(const gwb_ham* h) {
  static const bool env_on = [] {
    const char* v = std::getenv("GWB_TC_NONLOCAL");
    return !(v && v[0] == '0');
  }();
  return env_on && h->nproj >= TC_NONLOCAL_MIN_NPROJ;
}

// out += P^T D (P^* . c) with split-BF16 tensor-core products:
// becp = c P^H (A B^H, FP32 accumulation, float64 slice sums), bd = becp D in
// float64 written as BF16 planes, out += bd P (A B, P read MN-major). The
// BF16 planes of P are built once per set of projectors.
static int nonlocal_tc(gwb_ham* h, const cplx<double>* c, int64_t ck, cplx<double>* out, int64_t ok, int nb,
                       cudaStream_t st) {
  const int nk = h->nk, np = h->nproj, npw = h->npw_max;
  const int64_t ldp = ((int64_t)npw + 7) / 8 * 8, ldq = ((int64_t)np + 7) / 8 * 8;
  int rc;
  if (!h->d_tcstatus) {
    size_t n = 0;
    if ((rc = ensure_buf(h, (void**)&h->d_tcstatus, &n, sizeof(int)))) return rc;
    GWB_CUDA_TRY(cudaMemsetAsync(h->d_tcstatus, 0, sizeof(int), st));
  }
  if (!h->pplanes_ok) {
    if ((rc = ensure_buf(h, &h->d_pplanes, &h->pplanes_bytes, (size_t)nk * 4 * np * ldp * 2))) return rc;
    if ((rc = gwb_tc_planes(nk, np, npw, h->d_p64, npw, (int64_t)np * npw, GWB_C128, 0, h->d_pplanes, ldp, np, 0,
                            st)))
      return rc;
    h->pplanes_ok = true;
  }
  if ((rc = ensure_buf(h, &h->d_cplanes, &h->cplanes_bytes, (size_t)nk * 4 * nb * ldp * 2))) return rc;
  if ((rc = ensure_buf(h, &h->d_becp, &h->becp_bytes, (size_t)nk * nb * np * 16))) return rc;
  if ((rc = ensure_buf(h, &h->d_bdplanes, &h->bdplanes_bytes, (size_t)nk * 4 * nb * ldq * 2))) return rc;
  const int64_t wb = gwb_zgemm_tc_work_bytes(2, nb, np, npw, nk);
  if (wb > 0 && (rc = ensure_buf(h, &h->d_tcwork, &h->tcwork_bytes, (size_t)wb))) return rc;
  if ((rc = gwb_tc_planes(nk, nb, npw, c, npw, ck, GWB_C128, 0, h->d_cplanes, ldp, nb, 0, st))) return rc;
  if ((rc = gwb_zgemm_tc(2, nb, np, npw, 1.0, 0.0, h->d_cplanes, ldp, nb, h->d_pplanes, ldp, np, 0.0, 0.0, h->d_becp,
                         np, (int64_t)nb * np, nk, h->d_tcwork, h->tcwork_bytes, h->d_tcstatus, st)))
    return rc;
  if ((rc = tc_becp_d_planes(nk, nb, np, (const cplx<double>*)h->d_becp, h->d_d64, h->d_cols, h->d_bdplanes, ldq,
                             st)))
    return rc;
  return gwb_zgemm_tc(0, nb, npw, np, 1.0, 0.0, h->d_bdplanes, ldq, nb, h->d_pplanes, ldp, np, 1.0, 0.0, out, npw, ok,
                      nk, nullptr, 0, h->d_tcstatus, st);
}

// out = T c + local(c): the kinetic and FFT local terms, in chunks of bands.
template <typename T, typename SIO>
static int local_term(gwb_ham* h, const SIO* c, int64_t ck, SIO* out, int64_t ok, int nb, cudaStream_t st) {
  int nbc = 0;
  const int rc = chunk_scratch(h, nb, sizeof(cplx<T>), &nbc);
  if (rc) return rc;
  FftRun<T> f = fft_run<T>(h, nbc);
  f.c = c, f.out = out, f.ck = ck, f.ok = ok;
  f.io64 = sizeof(SIO) == 16;
  for (int b0 = 0; b0 < nb; b0 += nbc) {
    f.b0 = b0;
    f.nbc = std::min(nbc, nb - b0);
    place_rows(h, &f);
    GWB_CUDA_TRY(fft_rows_inverse(f, st));
    GWB_CUDA_TRY(fft_cols_inverse(f, st));
    GWB_CUDA_TRY(fft_pencil_vloc(f, st));
    GWB_CUDA_TRY(fft_cols_forward(f, st));
    GWB_CUDA_TRY(fft_rows_forward(f, st));
    count_launches(5);
  }
  if (h->ndup) {
    k_duplicate_slots<T, SIO><<<std::min(148 * 4, (h->ndup * nb + 255) / 256), 256, 0, st>>>(
        h->d_dup, h->ndup, c, ck, out, ok, f.t, nb, h->npw_max);
    GWB_LAUNCH_CHECK();
    count_launches(1);
  }
  return GWB_OK;
}

// float64 arithmetic on complex128 rows: the float64 tensor instruction
// (zmma.cuh); anything else the CUDA-core kernels above. Measured with 256
// projectors, 2 k x 129 bands x 37,000 plane waves: becp 1908 -> 920 us, update
// 1369 -> 750 us.
template <typename T, typename SIO>
constexpr bool nl_zmma = std::is_same<T, double>::value && std::is_same<SIO, cplx<double>>::value;

// becp partial sums over G slices into d_part (slice, k, band, projector).
template <typename T, typename SIO>
static int becp_slices(gwb_ham* h, const SIO* c, int64_t ck, int nb, int* nsl, cudaStream_t st) {
  const size_t es = sizeof(cplx<T>);
  const int npw = h->npw_max, np = h->nproj;
  int gslice = 0;
  if constexpr (nl_zmma<T, SIO>) {
    *nsl = zmma_nh_slices(nb, np, npw, h->nk, npw, h->nl_target > 0 ? h->nl_target : 4 * 148, &gslice);
  } else {
    const int ns = nl_slices(h, nb);
    gslice = ((npw + ns - 1) / ns + NL_TG - 1) / NL_TG * NL_TG;
    *nsl = (npw + gslice - 1) / gslice;
  }
  int rc = ensure_buf(h, &h->d_part, &h->part_bytes, (size_t)*nsl * h->nk * nb * np * es);
  if (rc) return rc;
  if ((rc = ensure_buf(h, &h->d_bd, &h->bd_bytes, (size_t)h->nk * nb * np * es))) return rc;
  if constexpr (nl_zmma<T, SIO>) {
    GWB_CUDA_TRY(zmma_nh(nb, np, npw, gslice, *nsl, c, npw, ck, h->d_p64, npw, (int64_t)np * npw,
                         (cplx<double>*)h->d_part, h->nk, st));
  } else {
    const cplx<T>* P = sizeof(T) == 8 ? (const cplx<T>*)h->d_p64 : (const cplx<T>*)h->d_p32;
    dim3 g4((np + NL_TP - 1) / NL_TP, (nb + NL_TB - 1) / NL_TB, h->nk * *nsl);
    GWB_CUDA_TRY(launch_chained(k_becp_partial<T, SIO>, g4, 256, 0, st, c, P, (cplx<T>*)h->d_part, h->nk, nb, np, npw,
                                gslice, ck));
  }
  count_launches(1);
  return GWB_OK;
}

template <typename T, typename SIO>
static int apply_impl(gwb_ham* h, const SIO* c, int64_t ck, SIO* out, int64_t ok, int nb, cudaStream_t st) {
  const size_t es = sizeof(cplx<T>);
  const bool dbl = sizeof(T) == 8;
  int rc = local_term<T, SIO>(h, c, ck, out, ok, nb, st);
  if (rc) return rc;
  if constexpr (std::is_same<T, float>::value && std::is_same<SIO, cplx<double>>::value) {
    if (h->nproj > 0 && tc_nonlocal_enabled(h)) return nonlocal_tc(h, c, ck, out, ok, nb, st);
  }
  if (h->nproj > 0) {
    int nsl = 0;
    if ((rc = becp_slices<T, SIO>(h, c, ck, nb, &nsl, st))) return rc;
    const T* D = dbl ? (const T*)h->d_d64 : (const T*)h->d_d32;
    const int ngrp = std::max(1, 128 / h->nproj);
    GWB_CUDA_TRY(launch_chained(k_becp_reduce_d<T>, dim3(h->nk * nb), 128, (size_t)h->nproj * (1 + ngrp) * es, st,
                                (const cplx<T>*)h->d_part, D, h->d_cols, (cplx<T>*)h->d_bd, h->nk, nb, h->nproj, nsl));
    if constexpr (nl_zmma<T, SIO>) {
      GWB_CUDA_TRY(zmma_nn(nb, h->npw_max, h->nproj, (const cplx<double>*)h->d_bd, nullptr, h->d_p64, nullptr, 0, out,
                           ok, nullptr, 0, nullptr, h->nk, st));
    } else {
      const cplx<T>* P = dbl ? (const cplx<T>*)h->d_p64 : (const cplx<T>*)h->d_p32;
      dim3 g6((h->npw_max + 63) / 64, (nb + NL_TB - 1) / NL_TB, h->nk);
      GWB_CUDA_TRY(launch_chained(k_nl_add<T, SIO>, g6, 256, 0, st, (const cplx<T>*)h->d_bd, P, out, h->nk, nb, h->nproj,
                                  h->npw_max, ok));
    }
    count_launches(2);
  }
  return GWB_OK;
}

// Generalized apply: out_h = H c and out_s = S c = (c + sum_pq |p> q_pq <q|c>)
// masked, from one becp contraction.
template <typename T, typename SIO>
static int apply_hs_impl(gwb_ham* h, const SIO* c, int64_t ck, SIO* out_h, int64_t ohk, SIO* out_s, int64_t osk,
                         int nb, cudaStream_t st) {
  const size_t es = sizeof(cplx<T>);
  const bool dbl = sizeof(T) == 8;
  int rc = local_term<T, SIO>(h, c, ck, out_h, ohk, nb, st);
  if (rc) return rc;
  if (h->nproj > 0) {
    int nsl = 0;
    if ((rc = becp_slices<T, SIO>(h, c, ck, nb, &nsl, st))) return rc;
    if ((rc = ensure_buf(h, &h->d_bq, &h->bq_bytes, (size_t)h->nk * nb * h->nproj * es))) return rc;
    const T* D = dbl ? (const T*)h->d_d64 : (const T*)h->d_d32;
    const T* Q = dbl ? (const T*)h->d_q64 : (const T*)h->d_q32;
    const int ngrp = std::max(1, 128 / h->nproj);
    GWB_CUDA_TRY(launch_chained(k_becp_reduce_dq<T>, dim3(h->nk * nb), 128, (size_t)h->nproj * (1 + ngrp) * es, st,
                                (const cplx<T>*)h->d_part, D, h->d_cols, Q, h->q_cols, (cplx<T>*)h->d_bd,
                                (cplx<T>*)h->d_bq, h->nk, nb, h->nproj, nsl));
    count_launches(1);
  }
  if constexpr (nl_zmma<T, SIO>) {
    // with no projectors nothing is read from bq, but it still asks for S c = masked c
    const cplx<double>* bq = h->nproj > 0 ? (const cplx<double>*)h->d_bq : c;
    GWB_CUDA_TRY(zmma_nn(nb, h->npw_max, h->nproj, (const cplx<double>*)h->d_bd, bq, h->d_p64, c, ck, out_h, ohk, out_s,
                         osk, h->d_npw, h->nk, st));
  } else {
    const cplx<T>* P = dbl ? (const cplx<T>*)h->d_p64 : (const cplx<T>*)h->d_p32;
    dim3 g6((h->npw_max + 63) / 64, (nb + NL_TB - 1) / NL_TB, h->nk);
    GWB_CUDA_TRY(launch_chained(k_nl_add_hs<T, SIO>, g6, 256, 0, st, (const cplx<T>*)h->d_bd, (const cplx<T>*)h->d_bq, P,
                                c, ck, out_h, ohk, out_s, osk, h->d_npw, h->nk, nb, h->nproj, h->npw_max));
  }
  count_launches(1);
  return GWB_OK;
}

// Density of nb bands (float64 FFTs): axes 2 and 1 of a band chunk into W, then
// the pencil kernel accumulating w |psi|^2 per k and band group, finally their sum.
template <typename SIO>
static int density_impl(gwb_ham* h, const SIO* c, int64_t ck, int nb, const double* w, int64_t wk, double scale,
                        double* rho, cudaStream_t st) {
  const FftGeom& g = h->g;
  const size_t N = (size_t)g.n[0] * g.n[1] * g.n[2];
  int nbc = 0;
  int rc = chunk_scratch(h, nb, sizeof(cplx<double>), &nbc);
  if (rc) return rc;
  // band groups: about 8 blocks of 16 pencils per SM, at least two bands each;
  // the same for every chunking, so that chunks do not change the sums
  const int64_t blocks = (int64_t)h->nk * ((g.n[1] * g.n[2] + 15) / 16);
  const int ngrp = (int)std::max<int64_t>(1, std::min<int64_t>((8 * 148 + blocks - 1) / blocks, nb / 2));
  rc = ensure_buf(h, (void**)&h->d_rhok, &h->rhok_bytes, (size_t)h->nk * ngrp * N * sizeof(double));
  if (rc) return rc;
  FftRun<double> f = fft_run<double>(h, nbc);
  f.c = c, f.ck = ck, f.io64 = sizeof(SIO) == 16;
  f.w = w, f.wk = wk, f.rho = h->d_rhok, f.ngrp = ngrp;
  for (int b0 = 0; b0 < nb; b0 += nbc) {
    f.b0 = b0;
    f.nbc = std::min(nbc, nb - b0);
    f.first = b0 == 0;
    place_rows(h, &f);
    GWB_CUDA_TRY(fft_rows_inverse(f, st));
    GWB_CUDA_TRY(fft_cols_inverse(f, st));
    GWB_CUDA_TRY(fft_pencil_density(f, st));
    count_launches(3);
  }
  const int sum_blocks = (int)std::min<size_t>((N + 255) / 256, 148 * 8);
  k_density_sum<<<sum_blocks, 256, 0, st>>>(h->nk * ngrp, (int64_t)N, h->d_rhok, scale, rho);
  GWB_LAUNCH_CHECK();
  count_launches(1);
  return GWB_OK;
}
}  // namespace gwb

using namespace gwb;

extern "C" {

const char* gwb_last_error(void) { return g_last_error.c_str(); }
const char* gwb_version(void) { return "gwb 0.1 sm_100a"; }
unsigned long long gwb_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

static int create_handle(const gwb_ham_geometry* geom, int device, gwb_ham** out) {
  GWB_REQUIRE(geom && out, "null argument");
  GWB_REQUIRE(geom->nk > 0 && geom->npw_max > 0 && geom->nproj >= 0, "bad nk/npw_max/nproj");
  GWB_REQUIRE(geom->npw && geom->flat_idx, "null npw/flat_idx");
  *out = nullptr;
  std::unique_ptr<gwb_ham, int (*)(gwb_ham*)> owner(new gwb_ham(), gwb_ham_destroy);  // also where host memory runs out
  gwb_ham* h = owner.get();
  h->device = device;
  h->nk = geom->nk;
  h->npw_max = geom->npw_max;
  h->nproj = geom->nproj;
  FftGeom& g = h->g;
  for (int a = 0; a < 3; ++a) {
    g.n[a] = geom->n[a];
    if (!axis_ok(g.n[a])) {
      set_error("FFT axis length " + std::to_string(geom->n[a]) + " unsupported (need <=128, factors 2,3,5,7)");
      return GWB_ERR_ARG;
    }
  }
  const int n0 = g.n[0], n1 = g.n[1], n2 = g.n[2];
  const int64_t nbox = (int64_t)n0 * n1 * n2;
  h->npw_host.assign(geom->npw, geom->npw + geom->nk);
  // box coordinates of every sphere point, Miller extents over all k
  struct Cell {
    uint8_t i0, i1, i2;
  };
  std::vector<size_t> first(h->nk + 1, 0);  // k's points in cell (the padding takes no host memory)
  for (int k = 0; k < h->nk; ++k) {
    const int64_t np_k = h->npw_host[k];
    if (np_k < 0 || np_k > h->npw_max) {
      set_error("npw[k] out of range");
      return GWB_ERR_ARG;
    }
    first[k + 1] = first[k] + np_k;
  }
  std::vector<Cell> cell(first[h->nk]);
  int M[3] = {0, 0, 0};
  for (int k = 0; k < h->nk; ++k) {
    for (int64_t gi = 0; gi < h->npw_host[k]; ++gi) {
      const int64_t f = geom->flat_idx[(size_t)k * h->npw_max + gi];
      if (f < 0 || f >= nbox) {
        set_error("flat_idx out of the box");
        return GWB_ERR_ARG;
      }
      const unsigned u = (unsigned)f, q = u / (unsigned)n2, i0 = q / (unsigned)n1;
      const int idx[3] = {(int)i0, (int)(q - i0 * n1), (int)(u - q * n2)};
      cell[first[k] + gi] = {(uint8_t)idx[0], (uint8_t)idx[1], (uint8_t)idx[2]};
      for (int a = 0; a < 3; ++a) {
        const int m = idx[a] <= g.n[a] / 2 ? idx[a] : idx[a] - g.n[a];
        M[a] = std::max(M[a], std::abs(m));
      }
    }
  }
  for (int a = 0; a < 3; ++a) {
    g.L[a] = std::min(2 * M[a] + 1, g.n[a]);
    g.M[a] = g.L[a] == g.n[a] ? g.n[a] : M[a];
  }
  const int L0 = g.L[0];
  // row slots of the occupied (j0, i1) of each k, and the sphere index of each row point
  auto compact0 = [&](int i0) -> int { return g.L[0] == n0 || i0 <= g.M[0] ? i0 : i0 - (n0 - L0); };
  std::vector<int> rowof((size_t)h->nk * L0 * n1, -1);
  std::vector<int> nrow_k(h->nk, 0);
  for (int k = 0; k < h->nk; ++k) {
    int* ro = rowof.data() + (size_t)k * L0 * n1;
    const Cell* ck = cell.data() + first[k];
    for (int64_t gi = 0; gi < h->npw_host[k]; ++gi) ro[compact0(ck[gi].i0) * n1 + ck[gi].i1] = 0;
    for (int i = 0; i < L0 * n1; ++i)
      if (ro[i] == 0) ro[i] = nrow_k[k]++;
  }
  g.nrow = std::max(1, *std::max_element(nrow_k.begin(), nrow_k.end()));
  std::vector<int> map((size_t)h->nk * g.nrow * n2, -1), dup;
  for (int k = 0; k < h->nk; ++k)
    for (int64_t gi = h->npw_host[k] - 1; gi >= 0; --gi) {
      const Cell p = cell[first[k] + gi];
      const int row = rowof[((size_t)k * L0 + compact0(p.i0)) * n1 + p.i1];
      int& slot = map[((size_t)k * g.nrow + row) * n2 + p.i2];
      if (slot < 0) slot = (int)gi;
      else dup.insert(dup.end(), {k, (int)gi, slot});
    }
  h->ndup = (int)(dup.size() / 3);
  std::vector<int> npw32(h->npw_host.begin(), h->npw_host.end());
  // twiddles exp(-2 pi i a k / n) at k R2 + a (n = R1 R2)
  std::vector<cplx<double>> tw64[3];
  std::vector<cplx<float>> tw32[3];
  for (int a = 0; a < 3; ++a) {
    const int n = g.n[a], R2 = n / fft_r1(n);
    for (int t = 0; t < n; ++t) {
      const cplx<double> w = conj(unit_root((t / R2) * (t % R2), n));
      tw64[a].push_back(w);
      tw32[a].push_back(mk<float>((float)w.x, (float)w.y));
    }
  }
  auto fail = [&](cudaError_t e) {
    cudaGetLastError();
    set_error(std::string("gwb_ham_create: ") + cudaGetErrorString(e));
    return GWB_ERR_CUDA;
  };
  auto no_room = [&] { return fail(cudaErrorMemoryAllocation); };
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return fail(e);
#define GWB_ALLOC_COPY(dst, vec)                                                            \
  do {                                                                                      \
    if (!g_pool.alloc(device, (void**)&(dst), (vec).size() * sizeof((vec)[0]))) return no_room(); \
    e = cudaMemcpy((dst), (vec).data(), (vec).size() * sizeof((vec)[0]), cudaMemcpyHostToDevice); \
    if (e != cudaSuccess) return fail(e);                                                   \
  } while (0)
  GWB_ALLOC_COPY(h->d_map, map);
  GWB_ALLOC_COPY(h->d_rowof, rowof);
  if (h->ndup) GWB_ALLOC_COPY(h->d_dup, dup);
  GWB_ALLOC_COPY(h->d_npw, npw32);
  for (int a = 0; a < 3; ++a) {
    GWB_ALLOC_COPY(h->d_tw64[a], tw64[a]);
    GWB_ALLOC_COPY(h->d_tw32[a], tw32[a]);
  }
#undef GWB_ALLOC_COPY
  const size_t nkp = (size_t)h->nk * h->npw_max;
  if (!g_pool.alloc(device, (void**)&h->d_t64, nkp * 8)) return no_room();
  if (!g_pool.alloc(device, (void**)&h->d_t32, nkp * 4)) return no_room();
  if (!g_pool.alloc(device, (void**)&h->d_v64, nbox * 8)) return no_room();
  if (!g_pool.alloc(device, (void**)&h->d_v32, nbox * 4)) return no_room();
  if (h->nproj > 0) {
    const size_t np = (size_t)h->nk * h->nproj * h->npw_max;
    if (!g_pool.alloc(device, (void**)&h->d_p64, np * 16)) return no_room();
    if (!g_pool.alloc(device, (void**)&h->d_p32, np * 8)) return no_room();
    if (!g_pool.alloc(device, (void**)&h->d_d64, (size_t)h->nproj * h->nproj * 8)) return no_room();
    if (!g_pool.alloc(device, (void**)&h->d_d32, (size_t)h->nproj * h->nproj * 4)) return no_room();
    if (!g_pool.alloc(device, (void**)&h->d_cols.cnt, (size_t)h->nproj * sizeof(int))) return no_room();
    if (!g_pool.alloc(device, (void**)&h->d_cols.idx, (size_t)h->nproj * h->nproj * sizeof(int))) return no_room();
  }
  g_pool.handles(device, 1);
  h->counted = true;
  *out = owner.release();
  return GWB_OK;
}

int gwb_ham_create(const gwb_ham_geometry* geom, int device, gwb_ham** out) {
  try {
    return create_handle(geom, device, out);
  } catch (const std::bad_alloc&) {
    set_error("gwb_ham_create: out of host memory");
    return GWB_ERR_ALLOC;
  }
}

int gwb_ham_destroy(gwb_ham* h) {
  if (!h) return GWB_OK;
  if (h->W.p) {
    // the scratch may serve the next handle once nothing in flight uses it
    int cur = 0;
    const bool idle = cudaGetDevice(&cur) == cudaSuccess && cudaSetDevice(h->device) == cudaSuccess &&
                      cudaDeviceSynchronize() == cudaSuccess;
    if (idle) {
      g_pool.give(h->device, h->W.p, h->W.bytes);
      h->W = {};
    } else {
      cudaGetLastError();
    }
    cudaSetDevice(cur);
  }
  if (h->counted) g_pool.handles(h->device, -1);
  void* ptrs[] = {h->d_npw, h->d_map, h->d_rowof, h->d_dup, h->d_t64, h->d_t32, h->d_v64,
                  h->d_v32, h->d_p64, h->d_p32, h->d_d64, h->d_d32, h->d_q64, h->d_q32, h->d_cols.cnt, h->d_cols.idx,
                  h->q_cols.cnt, h->q_cols.idx, h->W.p, h->d_part, h->d_bd, h->d_bq,
                  h->d_pplanes, h->d_cplanes, h->d_becp, h->d_bdplanes, h->d_tcwork, h->d_tcstatus, h->d_rhok,
                  h->d_tw64[0], h->d_tw64[1], h->d_tw64[2], h->d_tw32[0], h->d_tw32[1], h->d_tw32[2]};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  delete h;
  return GWB_OK;
}

static unsigned blocks_for(size_t n, unsigned bs) { return (unsigned)((n + bs - 1) / bs); }

int gwb_ham_set_kinetic(gwb_ham* h, const double* t, void* stream) {
  GWB_REQUIRE(h && t, "null argument");
  cudaStream_t st = (cudaStream_t)stream;
  const size_t n = (size_t)h->nk * h->npw_max;
  GWB_CUDA_TRY(cudaMemcpyAsync(h->d_t64, t, n * 8, cudaMemcpyDeviceToDevice, st));
  k_scale_copy<float><<<blocks_for(n, 256), 256, 0, st>>>(t, h->d_t32, n, 1.0);
  GWB_LAUNCH_CHECK();
  h->have_t = true;
  return GWB_OK;
}

int gwb_ham_set_potential(gwb_ham* h, const double* v, void* stream) {
  GWB_REQUIRE(h && v, "null argument");
  cudaStream_t st = (cudaStream_t)stream;
  const size_t n = (size_t)h->g.n[0] * h->g.n[1] * h->g.n[2];
  const double s = 1.0 / (double)n;
  k_scale_copy<double><<<blocks_for(n, 256), 256, 0, st>>>(v, h->d_v64, n, s);
  k_scale_copy<float><<<blocks_for(n, 256), 256, 0, st>>>(v, h->d_v32, n, s);
  GWB_LAUNCH_CHECK();
  h->have_v = true;
  return GWB_OK;
}

int gwb_ham_set_projectors(gwb_ham* h, const void* p, const double* dij, void* stream) {
  GWB_REQUIRE(h, "null handle");
  if (h->nproj == 0) {
    h->have_p = true;
    return GWB_OK;
  }
  GWB_REQUIRE(p && dij, "null projector pointer");
  cudaStream_t st = (cudaStream_t)stream;
  const size_t np = (size_t)h->nk * h->nproj * h->npw_max;
  const size_t nd = (size_t)h->nproj * h->nproj;
  GWB_CUDA_TRY(cudaMemcpyAsync(h->d_p64, p, np * 16, cudaMemcpyDeviceToDevice, st));
  k_c128_to_c64<<<blocks_for(np, 256), 256, 0, st>>>((const cplx<double>*)p, h->d_p32, np);
  GWB_CUDA_TRY(cudaMemcpyAsync(h->d_d64, dij, nd * 8, cudaMemcpyDeviceToDevice, st));
  h->pplanes_ok = false;  // the tensor-core planes of P are rebuilt on next use
  k_scale_copy<float><<<blocks_for(nd, 256), 256, 0, st>>>(dij, h->d_d32, nd, 1.0);
  k_column_lists<<<blocks_for(h->nproj, 64), 64, 0, st>>>(dij, h->nproj, h->d_cols.cnt, h->d_cols.idx);
  GWB_LAUNCH_CHECK();
  h->have_p = true;
  return GWB_OK;
}

int gwb_ham_apply_strided(gwb_ham* h, const void* c, int64_t c_kstride, void* out, int64_t out_kstride,
                          int32_t nb, int32_t io_dtype, int32_t prec, void* stream) {
  GWB_REQUIRE(h && c && out, "null argument");
  GWB_REQUIRE(nb >= 0, "nb < 0");
  GWB_REQUIRE(h->have_t && h->have_v && h->have_p, "kinetic, potential and projectors must be set first");
  GWB_REQUIRE(io_dtype == GWB_C64 || io_dtype == GWB_C128, "io_dtype must be GWB_C64 or GWB_C128");
  GWB_REQUIRE(prec == GWB_FP32 || prec == GWB_FP64, "prec must be GWB_FP32 or GWB_FP64");
  GWB_REQUIRE(c != out, "c and out must not overlap");
  GWB_REQUIRE(c_kstride >= (int64_t)nb * h->npw_max && out_kstride >= (int64_t)nb * h->npw_max,
              "k stride smaller than nb * npw_max");
  if (nb == 0) return GWB_OK;
  cudaError_t e = cudaSetDevice(h->device);
  if (e != cudaSuccess) {
    set_error(cudaGetErrorString(e));
    return GWB_ERR_CUDA;
  }
  cudaStream_t st = (cudaStream_t)stream;
  if (io_dtype == GWB_C128) {
    auto* ci = (const cplx<double>*)c;
    auto* co = (cplx<double>*)out;
    return prec == GWB_FP64 ? apply_impl<double>(h, ci, c_kstride, co, out_kstride, nb, st)
                            : apply_impl<float>(h, ci, c_kstride, co, out_kstride, nb, st);
  }
  auto* ci = (const cplx<float>*)c;
  auto* co = (cplx<float>*)out;
  return prec == GWB_FP64 ? apply_impl<double>(h, ci, c_kstride, co, out_kstride, nb, st)
                          : apply_impl<float>(h, ci, c_kstride, co, out_kstride, nb, st);
}

int gwb_ham_apply(gwb_ham* h, const void* c, void* out, int32_t nb, int32_t io_dtype, int32_t prec,
                  void* stream) {
  GWB_REQUIRE(h, "null handle");
  const int64_t ks = (int64_t)nb * h->npw_max;
  return gwb_ham_apply_strided(h, c, ks, out, ks, nb, io_dtype, prec, stream);
}

int gwb_ham_set_tuning(gwb_ham* h, int64_t w_budget_bytes, int32_t nl_target_ctas) {
  GWB_REQUIRE(h, "null handle");
  GWB_REQUIRE(w_budget_bytes >= 0 && nl_target_ctas >= 0, "tuning values must be >= 0");
  h->w_budget = (size_t)w_budget_bytes;
  h->W.denied = SIZE_MAX;
  h->nl_target = nl_target_ctas;
  return GWB_OK;
}

int gwb_ham_set_fft_threads(gwb_ham* h, int32_t threads_fp32, int32_t threads_fp64) {
  GWB_REQUIRE(h, "null handle");
  auto ok = [](int32_t n) { return n == 0 || n == 256 || n == 512 || n == 1024; };
  GWB_REQUIRE(ok(threads_fp32) && ok(threads_fp64), "FFT block threads must be 0, 256, 512 or 1024");
  return GWB_OK;  // a hint: the block sizes of the FFT kernels follow from the axis lengths
}

int gwb_ham_set_overlap(gwb_ham* h, const double* q, void* stream) {
  GWB_REQUIRE(h, "null handle");
  GWB_REQUIRE(h->have_p, "projectors must be set before the overlap");
  if (h->nproj == 0) {
    h->have_q = true;
    return GWB_OK;
  }
  GWB_REQUIRE(q, "null overlap pointer");
  GWB_CUDA_TRY(cudaSetDevice(h->device));
  cudaStream_t st = (cudaStream_t)stream;
  const size_t nd = (size_t)h->nproj * h->nproj;
  if (!h->d_q64) {
    // all of the tables or none: a later call must not find some of them
    if (!g_pool.alloc_all(h->device, {{(void**)&h->d_q64, nd * 8},
                                      {(void**)&h->d_q32, nd * 4},
                                      {(void**)&h->q_cols.cnt, (size_t)h->nproj * sizeof(int)},
                                      {(void**)&h->q_cols.idx, nd * sizeof(int)}})) {
      set_error("device allocation of the overlap tables failed");
      return GWB_ERR_CUDA;
    }
  }
  GWB_CUDA_TRY(cudaMemcpyAsync(h->d_q64, q, nd * 8, cudaMemcpyDeviceToDevice, st));
  k_scale_copy<float><<<blocks_for(nd, 256), 256, 0, st>>>(q, h->d_q32, nd, 1.0);
  k_column_lists<<<blocks_for(h->nproj, 64), 64, 0, st>>>(q, h->nproj, h->q_cols.cnt, h->q_cols.idx);
  GWB_LAUNCH_CHECK();
  h->have_q = true;
  return GWB_OK;
}

int gwb_ham_apply_hs(gwb_ham* h, const void* c, int64_t c_kstride, void* out_h, int64_t oh_kstride, void* out_s,
                     int64_t os_kstride, int32_t nb, int32_t io_dtype, int32_t prec, void* stream) {
  GWB_REQUIRE(h && c && out_h && out_s, "null argument");
  GWB_REQUIRE(nb >= 0, "nb < 0");
  GWB_REQUIRE(h->have_t && h->have_v && h->have_p, "kinetic, potential and projectors must be set first");
  GWB_REQUIRE(h->have_q, "the overlap (gwb_ham_set_overlap) must be set first");
  GWB_REQUIRE(io_dtype == GWB_C64 || io_dtype == GWB_C128, "io_dtype must be GWB_C64 or GWB_C128");
  GWB_REQUIRE(prec == GWB_FP32 || prec == GWB_FP64, "prec must be GWB_FP32 or GWB_FP64");
  GWB_REQUIRE(c != out_h && c != out_s && out_h != out_s, "c, out_h and out_s must not overlap");
  const int64_t row = (int64_t)nb * h->npw_max;
  GWB_REQUIRE(c_kstride >= row && oh_kstride >= row && os_kstride >= row, "k stride smaller than nb * npw_max");
  if (nb == 0) return GWB_OK;
  GWB_CUDA_TRY(cudaSetDevice(h->device));
  cudaStream_t st = (cudaStream_t)stream;
  if (io_dtype == GWB_C128) {
    auto* ci = (const cplx<double>*)c;
    auto* oh = (cplx<double>*)out_h;
    auto* os = (cplx<double>*)out_s;
    return prec == GWB_FP64 ? apply_hs_impl<double>(h, ci, c_kstride, oh, oh_kstride, os, os_kstride, nb, st)
                            : apply_hs_impl<float>(h, ci, c_kstride, oh, oh_kstride, os, os_kstride, nb, st);
  }
  auto* ci = (const cplx<float>*)c;
  auto* oh = (cplx<float>*)out_h;
  auto* os = (cplx<float>*)out_s;
  return prec == GWB_FP64 ? apply_hs_impl<double>(h, ci, c_kstride, oh, oh_kstride, os, os_kstride, nb, st)
                          : apply_hs_impl<float>(h, ci, c_kstride, oh, oh_kstride, os, os_kstride, nb, st);
}

int gwb_ham_density(gwb_ham* h, const void* c, int64_t c_kstride, int32_t nb, int32_t io_dtype,
                    const double* weights, int64_t w_kstride, double scale, double* rho, void* stream) {
  GWB_REQUIRE(h && c && weights && rho, "null argument");
  GWB_REQUIRE(nb > 0, "nb must be positive");
  GWB_REQUIRE(io_dtype == GWB_C64 || io_dtype == GWB_C128, "io_dtype must be GWB_C64 or GWB_C128");
  GWB_REQUIRE(c_kstride >= (int64_t)nb * h->npw_max, "k stride smaller than nb * npw_max");
  GWB_REQUIRE(w_kstride >= nb, "weight k stride smaller than nb");
  GWB_CUDA_TRY(cudaSetDevice(h->device));
  cudaStream_t st = (cudaStream_t)stream;
  if (io_dtype == GWB_C128)
    return density_impl(h, (const cplx<double>*)c, c_kstride, nb, weights, w_kstride, scale, rho, st);
  return density_impl(h, (const cplx<float>*)c, c_kstride, nb, weights, w_kstride, scale, rho, st);
}

size_t gwb_ham_scratch_bytes(const gwb_ham* h) {
  return h ? h->W.bytes + h->part_bytes + h->bd_bytes + h->bq_bytes + h->pplanes_bytes + h->cplanes_bytes + h->becp_bytes +
                 h->bdplanes_bytes + h->tcwork_bytes + h->rhok_bytes
           : 0;
}

int gwb_ham_tc_status(gwb_ham* h, int* status) {
  GWB_REQUIRE(h && status, "null argument");
  *status = 0;
  if (!h->d_tcstatus) return GWB_OK;
  GWB_CUDA_TRY(cudaSetDevice(h->device));
  GWB_CUDA_TRY(cudaMemcpy(status, h->d_tcstatus, sizeof(int), cudaMemcpyDeviceToHost));
  if (*status) {
    GWB_CUDA_TRY(cudaMemset(h->d_tcstatus, 0, sizeof(int)));
    set_error("tensor-core nonlocal term: a bounded pipeline wait ran out");
    return GWB_ERR_TIMEOUT;
  }
  return GWB_OK;
}

}  // extern "C"
