// Batched complex GEMM with row-major semantics over cuBLAS (the plain
// library GEMMs of the Davidson subspace steps).
//
// C[b] = alpha * op(A[b]) * op(B[b]) + beta * C[b], op in {N, T, H}, every
// matrix row-major with a leading dimension and a batch stride. A row-major
// matrix is the column-major storage of its transpose, so the call becomes
// C^T = op(B)^T op(A)^T in cuBLAS terms with the operands swapped.
#include <cublas_v2.h>

#include <algorithm>
#include <string>
#include <unordered_map>

#include "common.cuh"
#include "zmma.cuh"

namespace gwb {

// One cuBLAS handle per (host thread, device): a handle's stream is set before
// every call, so threads that drive solves on different streams at the same
// time must not share one.
static thread_local std::unordered_map<int, cublasHandle_t> g_blas;

int blas_handle(cublasHandle_t* out) {
  int dev = 0;
  GWB_CUDA_TRY(cudaGetDevice(&dev));
  auto it = g_blas.find(dev);
  if (it == g_blas.end()) {
    cublasHandle_t h;
    if (cublasCreate(&h) != CUBLAS_STATUS_SUCCESS) {
      set_error("cublasCreate failed");
      return GWB_ERR_CUDA;
    }
    it = g_blas.emplace(dev, h).first;
  }
  *out = it->second;
  return GWB_OK;
}

// Products of few rows against long ones that the own tiles (zmma_ab, launched in
// chain) take from cuBLAS. Measured, us own / cuBLAS, op(A) = A, batch 10 x N =
// 4625, 4 x 37000 and 1 x 750: 8 x 112: 18 / 31, 52 / 85, 6 / 8; 16 x 64: 21 / 21,
// 58 / 62, 6 / 7; 16 x 112: 34 / 33, 93 / 93, 8 / 8; 24 x 24: 14 / 20, 37 / 54, 6 /
// 19; 24 x 96: 37 / 41, 107 / 121, 10 / 19; 24 x 448: 151 / 159, 464 / 502, 40 / 17;
// 32 x 32: 20 / 21, 57 / 55, 6 / 14; 32 x 128: 65 / 58, 189 / 154, 17 / 9; 40 x 40:
// 34 / 37, 94 / 111, 6 / 16; 48 x 48: 40 / 39, 112 / 119; 64 x 64: 65 / 54, 182 /
// 156. The longer K, the more a cut per 8 terms costs, and one block per tile has
// the whole of K in sequence. 128 is past the native solver's bases (112); where
// the two are level its launches stay in chain.
static bool short_rows(int64_t M, int64_t N, int64_t K) {
  return N >= 8 * M && K <= (M <= 24 ? 128 : (M <= 40 ? M : 0));
}

static cublasOperation_t to_op(int op) {
  return op == 0 ? CUBLAS_OP_N : (op == 1 ? CUBLAS_OP_T : CUBLAS_OP_C);
}

}  // namespace gwb

using namespace gwb;

extern "C" int gwb_zgemm(int opA, int opB, int64_t M, int64_t N, int64_t K, double alpha_re, double alpha_im,
                         const void* A, int64_t lda, int64_t strideA, const void* B, int64_t ldb,
                         int64_t strideB, double beta_re, double beta_im, void* C, int64_t ldc,
                         int64_t strideC, int64_t batch, void* stream) {
  GWB_REQUIRE(opA >= 0 && opA <= 2 && opB >= 0 && opB <= 2, "op must be 0 (N), 1 (T) or 2 (H)");
  GWB_REQUIRE(M >= 0 && N >= 0 && K >= 0 && batch >= 0, "negative size");
  if (M == 0 || N == 0 || batch == 0) return GWB_OK;
  GWB_REQUIRE(A && B && C, "null matrix");
  // the solver's triangular transforms, projections and Ritz vectors of small blocks
  if (opB == 0 && opA <= 1 && K > 0 && batch <= 65535 && short_rows(M, N, K)) {
    GWB_REQUIRE(lda >= (opA ? M : K) && ldb >= N && ldc >= N, "leading dimension smaller than a row");  // as cuBLAS
    GWB_CUDA_TRY(zmma_ab(opA == 1, (int)M, (int)N, (int)K, mk<double>(alpha_re, alpha_im), (const cplx<double>*)A, lda,
                         strideA, (const cplx<double>*)B, ldb, strideB, mk<double>(beta_re, beta_im), (cplx<double>*)C,
                         ldc, strideC, (int)batch, (cudaStream_t)stream));
    count_launches(1);
    return GWB_OK;
  }
  cublasHandle_t h;
  int rc = blas_handle(&h);
  if (rc) return rc;
  if (cublasSetStream(h, (cudaStream_t)stream) != CUBLAS_STATUS_SUCCESS) {
    set_error("cublasSetStream failed");
    return GWB_ERR_CUDA;
  }
  const cuDoubleComplex alpha = make_cuDoubleComplex(alpha_re, alpha_im);
  const cuDoubleComplex beta = make_cuDoubleComplex(beta_re, beta_im);
  // row-major C (M x N) == column-major C^T (N x M) = op(B)^T op(A)^T
  cublasStatus_t s = cublasZgemmStridedBatched(
      h, to_op(opB), to_op(opA), (int)N, (int)M, (int)K, &alpha, (const cuDoubleComplex*)B, (int)ldb, strideB,
      (const cuDoubleComplex*)A, (int)lda, strideA, &beta, (cuDoubleComplex*)C, (int)ldc, strideC, (int)batch);
  if (s != CUBLAS_STATUS_SUCCESS) {
    set_error("cublasZgemmStridedBatched failed with status " + std::to_string((int)s));
    return GWB_ERR_CUDA;
  }
  return GWB_OK;
}

// ---------------------------------------------------------------------------
// Inner-product GEMM with a long reduction: C = alpha A B^H + beta C with
// A (M x K), B (N x K) row-major and M, N small (the subspace, projection and
// Gram products of the Davidson step: M, N <= a few hundred, K = npw). cuBLAS
// tiles such shapes into a few dozen CTAs; here K is split into slices so the
// grid fills the GPU, each CTA accumulates an output tile of one slice on the
// float64 tensor instruction (zmma.cuh), and a second kernel sums the slices in
// a fixed order (deterministic).
namespace gwb {

__global__ void k_zgemm_nh_reduce(int M, int N, int nslice, int batch, const cplx<double>* __restrict__ part,
                                  cplx<double> alpha, cplx<double> beta, cplx<double>* __restrict__ C, int64_t ldc,
                                  int64_t sC) {
  const int64_t total = (int64_t)batch * M * N;
  chain_wait();
  part = after_wait(part);
  C = after_wait(C);
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int b = (int)(idx / ((int64_t)M * N));
    const int64_t r = idx % ((int64_t)M * N);
    const int i = (int)(r / N), j = (int)(r % N);
    cplx<double> a = mk<double>(0.0, 0.0);
    for (int s = 0; s < nslice; ++s) a = a + part[(int64_t)s * total + idx];
    cplx<double>* c = C + b * sC + (int64_t)i * ldc + j;
    cplx<double> v = alpha * a;
    if (beta.x != 0.0 || beta.y != 0.0) v = v + beta * (*c);
    *c = v;
  }
}

}  // namespace gwb

extern "C" int gwb_zgemm_nh(int64_t M, int64_t N, int64_t K, double alpha_re, double alpha_im, const void* A,
                            int64_t lda, int64_t strideA, const void* B, int64_t ldb, int64_t strideB,
                            double beta_re, double beta_im, void* C, int64_t ldc, int64_t strideC, int64_t batch,
                            void* work, size_t work_bytes, void* stream) {
  GWB_REQUIRE(M >= 0 && N >= 0 && K >= 0 && batch >= 0, "negative size");
  if (M == 0 || N == 0 || batch == 0) return GWB_OK;
  GWB_REQUIRE(A && B && C && work, "null pointer");
  GWB_REQUIRE(M * N * batch * 16 <= (int64_t)work_bytes, "work smaller than one M*N*batch slice");
  const int64_t slice_bytes = M * N * batch * 16;
  int kslice = 0;
  const int ns = zmma_nh_slices((int)M, (int)N, (int)K, (int)batch, (int64_t)(work_bytes / slice_bytes), 4 * 148, &kslice);
  cudaStream_t st = (cudaStream_t)stream;
  GWB_CUDA_TRY(zmma_nh((int)M, (int)N, (int)K, kslice, ns, (const cplx<double>*)A, lda, strideA, (const cplx<double>*)B,
                       ldb, strideB, (cplx<double>*)work, (int)batch, st));
  const int64_t total = M * N * batch;
  const int blocks = (int)std::min<int64_t>((total + 255) / 256, 4096);
  GWB_CUDA_TRY(launch_chained(k_zgemm_nh_reduce, dim3(blocks), 256, 0, st, (int)M, (int)N, ns, (int)batch,
                              (const cplx<double>*)work, mk<double>(alpha_re, alpha_im), mk<double>(beta_re, beta_im),
                              (cplx<double>*)C, ldc, strideC));
  count_launches(2);
  return GWB_OK;
}
