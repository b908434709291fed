// Axis-0 kernels of the local term in float (fft_axis.cuh), one per axis length.
#include "fft_axis.cuh"

namespace gwb {

#define GWB_CASE(n) \
  case n: return fft_detail::launch_vloc<T, n>(f, st);
template <typename T> cudaError_t fft_pencil_vloc(const FftRun<T>& f, cudaStream_t st) {
  switch (f.n0) { GWB_FFT_LENGTHS(GWB_CASE) }
  return cudaErrorInvalidValue;
}
#undef GWB_CASE

template cudaError_t fft_pencil_vloc<float>(const FftRun<float>&, cudaStream_t);

}  // namespace gwb
