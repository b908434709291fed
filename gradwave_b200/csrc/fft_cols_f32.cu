// Axis-1 kernels of the local term in float (fft_axis.cuh), one per axis length.
#include "fft_axis.cuh"

namespace gwb {

#define GWB_CASE(n) \
  case n: return fft_detail::launch_cols<T, n>(k_cols_inverse<T, n>, f, st);
template <typename T> cudaError_t fft_cols_inverse(const FftRun<T>& f, cudaStream_t st) {
  switch (f.n1) { GWB_FFT_LENGTHS(GWB_CASE) }
  return cudaErrorInvalidValue;
}
#undef GWB_CASE

#define GWB_CASE(n) \
  case n: return fft_detail::launch_cols<T, n>(k_cols_forward<T, n>, f, st);
template <typename T> cudaError_t fft_cols_forward(const FftRun<T>& f, cudaStream_t st) {
  switch (f.n1) { GWB_FFT_LENGTHS(GWB_CASE) }
  return cudaErrorInvalidValue;
}
#undef GWB_CASE

template cudaError_t fft_cols_inverse<float>(const FftRun<float>&, cudaStream_t);
template cudaError_t fft_cols_forward<float>(const FftRun<float>&, cudaStream_t);

}  // namespace gwb
