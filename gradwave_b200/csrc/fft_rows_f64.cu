// Axis-2 kernels of the local term in double (fft_axis.cuh), one per axis length.
#include "fft_axis.cuh"

namespace gwb {

#define GWB_CASE(n) \
  case n: return fft_detail::launch_rows<T, n>(k_rows_inverse<T, n>, f, st);
template <typename T> cudaError_t fft_rows_inverse(const FftRun<T>& f, cudaStream_t st) {
  switch (f.n2) { GWB_FFT_LENGTHS(GWB_CASE) }
  return cudaErrorInvalidValue;
}
#undef GWB_CASE

#define GWB_CASE(n) \
  case n: return fft_detail::launch_rows<T, n>(k_rows_forward<T, n>, f, st);
template <typename T> cudaError_t fft_rows_forward(const FftRun<T>& f, cudaStream_t st) {
  switch (f.n2) { GWB_FFT_LENGTHS(GWB_CASE) }
  return cudaErrorInvalidValue;
}
#undef GWB_CASE

template cudaError_t fft_rows_inverse<double>(const FftRun<double>&, cudaStream_t);
template cudaError_t fft_rows_forward<double>(const FftRun<double>&, cudaStream_t);

}  // namespace gwb
