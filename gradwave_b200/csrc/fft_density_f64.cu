// Axis-0 kernels of the density (fft_axis.cuh), one per axis length.
#include "fft_axis.cuh"

namespace gwb {

#define GWB_CASE(n) \
  case n: return fft_detail::launch_density<double, n>(f, st);
cudaError_t fft_pencil_density(const FftRun<double>& f, cudaStream_t st) {
  switch (f.n0) { GWB_FFT_LENGTHS(GWB_CASE) }
  return cudaErrorInvalidValue;
}
#undef GWB_CASE

}  // namespace gwb
